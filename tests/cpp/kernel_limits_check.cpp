// Host-side check of kernel_limits.h: what is set or found for a kernel counts
// for one device only, a larger need is set again, and a failure is reported
// and not recorded.
#include <cstdio>

#include "kernel_limits.h"

using namespace hmb;

int main() {
    int a = 0, b = 0, calls = 0, fails = 0;
    KernelRecord r;
    auto expect = [&](int want, const char* what) {
        if (calls != want) {
            std::printf("fail %s: %d calls, expected %d\n", what, calls, want);
            ++fails;
        }
    };
    auto set = [&] { ++calls; };
    r.raise(0, &a, 49920, set);
    r.raise(0, &a, 49920, set);
    r.raise(0, &a, 100, set);
    expect(1, "one device");
    r.raise(1, &a, 49920, set);
    expect(2, "second device");
    r.raise(0, &b, 49920, set);
    expect(3, "second kernel");
    r.raise(1, &a, 60000, set);
    r.raise(1, &a, 50000, set);
    expect(4, "larger need");
    r.raise(0, &a, 49920, set);
    expect(4, "first device again");
    bool thrown = false;
    try {
        r.raise(2, &a, 1, [&] {
            ++calls;
            throw Error(HM_ERR_CUDA, "refused");
        });
    } catch (const Error&) {
        thrown = true;
    }
    if (!thrown) ++fails;
    r.raise(2, &a, 1, set);
    expect(6, "after a failure");
    KernelRecord q;
    calls = 0;
    auto find = [&] { return (size_t)(10 * ++calls); };
    if (q.get(0, &a, find) != 10 || q.get(0, &a, find) != 10 || q.get(1, &a, find) != 20 || calls != 2) {
        std::printf("fail occupancy record\n");
        ++fails;
    }
    if (fails) return 1;
    std::printf("ok\n");
    return 0;
}
