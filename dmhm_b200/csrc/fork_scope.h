// Launches on a context's side streams between a fork and a join: however the
// scope is left, the context's stream waits for what was queued on them, so
// that stream-ordered frees on it follow their kernels.
#pragma once

namespace hmb {

// Ctx: fork(mask) and join(mask) may throw; drain(mask) orders (or waits) without.
template <typename Ctx>
class ForkScope {
  public:
    // the side streams of a mask (0: nothing to do)
    ForkScope(Ctx& ctx, int mask) : ctx_(ctx), mask_(mask) {
        if (mask_ != 0) ctx_.fork(mask_);
    }
    ForkScope(const ForkScope&) = delete;
    ForkScope& operator=(const ForkScope&) = delete;
    void join() {
        if (mask_ != 0) ctx_.join(mask_);
        mask_ = 0;
    }
    ~ForkScope() {
        if (mask_ != 0) ctx_.drain(mask_);
    }

  private:
    Ctx& ctx_;
    int mask_;
};

}  // namespace hmb
