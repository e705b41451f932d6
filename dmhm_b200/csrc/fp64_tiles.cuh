// What the FP64 tensor-core kernels share: the 8 x 8 x 4 MMA and the
// asynchronous copies that stage its operands.
#pragma once

namespace hmb {

// d += a b, one 8 x 8 block: lane 4 g + t holds a(g, t), b(t, g), d(g, 2 t + h).
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Two doubles src[0], src[1] (`bytes` of them valid, zeros beyond) to the
// shared address d; `any` is a valid, 16-byte aligned address for copies of
// nothing.  No "memory" clobber: the destination is read only after
// cp_async_wait (which has one) and a barrier.
__device__ __forceinline__ void copy_pair(unsigned d, const double* src, int bytes, bool aligned,
                                          const double* any) {
    if (aligned) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(bytes ? src : any),
                     "r"(bytes));
    } else {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(bytes ? src : any),
                     "r"(bytes ? 8 : 0));
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d + 8),
                     "l"(bytes > 8 ? src + 1 : any), "r"(bytes > 8 ? 8 : 0));
    }
}

}  // namespace hmb
