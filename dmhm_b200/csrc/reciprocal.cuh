// The reflectors' reciprocal (round_reg.cuh).
#pragma once

namespace hmb {
namespace reground {

// 1 / x for a normal x whose reciprocal is normal: Newton's iteration
// y + y (1 - x y), which squares the relative error, from PTX's approximation
// (rcp.approx.ftz.f64, 20 bits), until the rounding of the last multiply-add is
// what is left: at most one unit in the last place (test_reciprocal_gpu.py).
// Every elimination step waits for it.  Inversion of 49 x 46 points (34 columns
// a block): 465 ms, with __drcp_rn 480, from an FP32 start 476; 64 x 64 points
// 299, 301 and 302.
__device__ __forceinline__ double reciprocal(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
#pragma unroll
    for (int i = 0; i < 3; ++i) y = fma(y, fma(-x, y, 1.0), y);
    return y;
}
__device__ __forceinline__ float reciprocal(float x) { return 1.0f / x; }

}  // namespace reground
}  // namespace hmb
