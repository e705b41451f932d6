// Launches on a context's side streams between a fork and a join: however the
// scope is left, the context's stream waits for what was queued on them, so
// that stream-ordered frees on it follow their kernels.
#pragma once

namespace hmb {

// Ctx: fork(n) and join(n) may throw; drain(n) orders (or waits) without.
template <typename Ctx>
class ForkScope {
  public:
    // n side streams (0: nothing to do)
    ForkScope(Ctx& ctx, int n) : ctx_(ctx), n_(n) {
        if (n_ > 0) ctx_.fork(n_);
    }
    ForkScope(const ForkScope&) = delete;
    ForkScope& operator=(const ForkScope&) = delete;
    void join() {
        if (n_ > 0) ctx_.join(n_);
        n_ = 0;
    }
    ~ForkScope() {
        if (n_ > 0) ctx_.drain(n_);
    }

  private:
    Ctx& ctx_;
    int n_;
};

}  // namespace hmb
