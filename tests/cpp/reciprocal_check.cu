// Device check of reciprocal.cuh against CUDA's correctly rounded reciprocal:
// the largest distance, in units of the last place of 1 / x, over random
// significands (and their ends) and exponents of -1000 to 1000, beyond what the
// square root of a sum of squares can be.
#include <cmath>
#include <cstdio>
#include <cuda_runtime.h>

#include "reciprocal.cuh"

__device__ unsigned long long mix(unsigned long long z) {
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

__device__ double ulps(double y, double x) {
    const double r = __drcp_rn(x);
    return fabs((double)(__double_as_longlong(y) - __double_as_longlong(r)));
}

__global__ void check(int n, double* worst) {
    double w = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const unsigned long long r = mix(2 * i + 1);
        const double m = i < 4 ? 1.0 + (i & 1 ? 0x1p-52 : 0.0) + (i & 2 ? 0.5 : 0.0)
                       : i < 6 ? 2.0 - 0x1p-52 * (i - 3) : 1.0 + (double)(r >> 12) * 0x1p-52;
        const int e = -1000 + (int)(mix(r) % 2001);
        const double sign = r & 1 ? -1.0 : 1.0, x = sign * scalbn(m, e);
        w = fmax(w, ulps(hmb::reground::reciprocal(x), x));
    }
    atomicMax(reinterpret_cast<unsigned long long*>(worst), __double_as_longlong(w));
}

int main() {
    double* d = nullptr;
    double w = -1.0;
    if (cudaMalloc(&d, sizeof(double)) != cudaSuccess || cudaMemset(d, 0, sizeof(double)) != cudaSuccess) return 2;
    check<<<296, 256>>>(1 << 22, d);
    if (cudaMemcpy(&w, d, sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    std::printf("%g\n", w);
    return 0;
}
