// Register-resident rounding: the same best rank-r approximation as do_round
// (lowrank.cu), organised so that its contractions run from registers.
//
// One CTA of NW warps owns one rounding.  In the QR phases a lane owns whole
// columns (column c = lane + 32 s) and a warp owns a slab of consecutive
// rows, so a column's part of a slab is an array of registers: a reflector is
// broadcast from shared memory and every lane takes its inner product and its
// update with plain multiply-adds, without shuffles.  A step's only
// communication is one barrier that adds the slabs' inner products.
//
// With A = U_s V_s^T (U_s, V_s the stacked factors) the steps are
//   1. R_v of V_s = Q_v R_v (Q_v itself is never needed),
//   2. T = U_s R_v^T, so that A A^T = T T^T (a dense block is its own T),
//   3. T P = Q_t R_1, Householder QR with column pivoting, stopped where the
//      remaining columns are rounding noise (k' reflectors are left),
//   4. R_1^T = Q_2 R_2, L = R_2^T (k' x k'): A and L have the same singular
//      values, and A's left singular vectors are Q_t times L's,
//   5. one-sided Jacobi on the columns of L: L W = Y S,
//   6. U_out = Q_t Y_r (orthonormal), V_out = A^T U_out = V_s (U_s^T U_out).
// Pivoting and the second triangularization make L nearly diagonal (Drmac and
// Veselic, SIAM J. Matrix Anal. Appl. 29, 2008): 2.5 to 4 sweeps where the
// core R_u R_v^T itself took 6 to 18, no rotation needs to be accumulated, and
// the columns cut in step 3 (a third of them on average) are never rotated.
// Bound: the chain of each elimination and rotation step (a reciprocal square
// root, a broadcast, one barrier: 700 to 900 cycles) times the 16 warps that
// fit an SM; the FP64 pipe is 20 % busy on 64 x 64 blocks, 14 % on 256 x 256.
// Measured, all roundings of one H*H product (do_round before): 64^2 grid, rank
// 16, 35,472 roundings 81.1 -> 16.0 ms; SchulzInvert there 1106 -> 237 ms in 28
// products; complex 24^2, rank 12, 924 -> 208 ms in 36; FP32, 72 x 68 grid, 765
// -> 192 ms in 28.
#pragma once

#include "fp64_tiles.cuh"
#include "reciprocal.cuh"
#include "round_sizing.h"

namespace hmb {
namespace reground {

constexpr int kMaxSweeps = 40;

template <typename R>
__device__ __forceinline__ R* shared_base() {
    extern __shared__ __align__(16) unsigned char round_dyn[];
    return reinterpret_cast<R*>(round_dyn);
}

// A thread's view of the CTA's shared memory.
template <typename R, int NW>
struct Cta {
    Layout L;
    int warp, lane;
    __device__ __forceinline__ R* us(int buf) const {
        return shared_base<R>() + (buf * NW + warp) * kSlabMax;
    }
    __device__ __forceinline__ R* part(int buf) const { return shared_base<R>() + L.part + buf * NW * L.cp; }
    __device__ __forceinline__ R* rowt(int buf) const { return shared_base<R>() + L.rowt + buf * L.cp; }
    __device__ __forceinline__ R* chunk(int buf) const {
        return shared_base<R>() + L.chunk + buf * NW * kChunk * L.rp;
    }
    __device__ __forceinline__ R* tau() const { return shared_base<R>() + L.tau; }
    __device__ __forceinline__ R* nrm() const { return shared_base<R>() + L.nrm; }
    __device__ __forceinline__ R* jex(int buf) const { return shared_base<R>() + L.jex + buf * NW * 32; }
    __device__ __forceinline__ R* mat() const { return shared_base<R>() + L.mat; }
    __device__ __forceinline__ int* flag() const { return reinterpret_cast<int*>(shared_base<R>() + L.order); }
    __device__ __forceinline__ int* order() const { return flag() + 1; }
};

// Two neighbouring values of shared memory in one access.
template <typename R> struct Pair;
template <> struct Pair<double> { using type = double2; };
template <> struct Pair<float> { using type = float2; };
template <typename R>
__device__ __forceinline__ typename Pair<R>::type load2(const R* p) {
    return *reinterpret_cast<const typename Pair<R>::type*>(p);
}

// A stack of columns: the first r2 from p2 scaled by s2, then r1 from p1
// scaled by s1.
struct Stack {
    const double* p1;
    const double* p2;
    double s1, s2;
    int rows, r1, r2, ld1, ld2;
    __device__ int cols() const { return r1 + r2; }
    __device__ const double* col(int c) const {
        return c < r2 ? p2 + (long long)c * ld2 : p1 + (long long)(c - r2) * ld1;
    }
    __device__ double scale(int c) const { return c < r2 ? s2 : s1; }
};

// Rows [row0, row0 + RPW) of a column of `rows` entries, scaled.
template <typename R, int RPW>
__device__ __forceinline__ void load_slab(R (&a)[RPW], const double* col, double scale, int row0,
                                          int rows, bool live) {
#pragma unroll
    for (int i = 0; i < RPW; ++i)
        a[i] = live && row0 + i < rows ? (R)(scale * col[row0 + i]) : R(0);
}

// The warp's slab of one column, fetched lane by lane (RPW <= 64: two rows a
// lane) and published to the warp through us.
template <typename R, int RPW>
struct Fetch {
    R v0, v1;
    __device__ __forceinline__ void get(const double* col, double scale, int row0, int rows,
                                        int lane) {
        v0 = lane < RPW && row0 + lane < rows ? (R)(scale * col[row0 + lane]) : R(0);
        if (RPW > 32)
            v1 = 32 + lane < RPW && row0 + 32 + lane < rows ? (R)(scale * col[row0 + 32 + lane]) : R(0);
    }
    __device__ __forceinline__ void put(R* us, int lane) const {
        if (lane < RPW) us[lane] = v0;
        if (RPW > 32 && 32 + lane < RPW) us[32 + lane] = v1;
        __syncwarp();
    }
};

// s[c] = sum over the slab of us[i] a[c][i]
template <typename R, int CPL, int RPW>
__device__ __forceinline__ void slab_dots(const R* us, const R (&a)[CPL][RPW], R (&s)[CPL]) {
    constexpr int NA = CPL == 1 ? 4 : 2;   // independent partial sums per column
    R t[CPL][NA];
#pragma unroll
    for (int c = 0; c < CPL; ++c)
#pragma unroll
        for (int q = 0; q < NA; ++q) t[c][q] = R(0);
#pragma unroll
    for (int i = 0; i < RPW; i += 2) {
        const auto u = load2(us + i);
#pragma unroll
        for (int c = 0; c < CPL; ++c) {
            t[c][i % NA] = r_fma(u.x, a[c][i], t[c][i % NA]);
            t[c][(i + 1) % NA] = r_fma(u.y, a[c][i + 1], t[c][(i + 1) % NA]);
        }
    }
#pragma unroll
    for (int c = 0; c < CPL; ++c) {
        s[c] = t[c][0] + t[c][1];
        if (NA == 4) s[c] += t[c][2] + t[c][3];
    }
}

template <typename R, int CPL, int RPW>
__device__ __forceinline__ void slab_axpy(const R* us, R (&a)[CPL][RPW], const R (&f)[CPL]) {
#pragma unroll
    for (int i = 0; i < RPW; i += 2) {
        const auto u = load2(us + i);
#pragma unroll
        for (int c = 0; c < CPL; ++c) {
            a[c][i] = r_fma(f[c], u.x, a[c][i]);
            a[c][i + 1] = r_fma(f[c], u.y, a[c][i + 1]);
        }
    }
}

// The same in the warp whose first row has just been finished: the remaining
// rows move up by one register as they are updated, so that its next row is
// again the first one and no register is addressed by a running index.
template <typename R, int CPL, int RPW>
__device__ __forceinline__ void slab_axpy_up(const R* us, R (&a)[CPL][RPW], const R (&f)[CPL]) {
#pragma unroll
    for (int i = 0; i < RPW; i += 2) {
        const auto u = load2(us + i);
#pragma unroll
        for (int c = 0; c < CPL; ++c) {
            if (i > 0) a[c][i - 1] = r_fma(f[c], u.x, a[c][i]);
            a[c][i] = r_fma(f[c], u.y, a[c][i + 1]);
        }
    }
#pragma unroll
    for (int c = 0; c < CPL; ++c) a[c][RPW - 1] = R(0);
}

// Column j (held by lane j % 32, slot j / 32) of the slab to us.
template <typename R, int CPL, int RPW>
__device__ __forceinline__ void publish_column(const R (&a)[CPL][RPW], int j, R* us, int lane) {
    const bool second = CPL > 1 && (j >> 5) == 1, third = CPL > 2 && (j >> 5) == 2;
    if (lane == (j & 31)) {
#pragma unroll
        for (int i = 0; i < RPW; i += 2) {
            typename Pair<R>::type v;
            v.x = a[0][i];
            v.y = a[0][i + 1];
            if constexpr (CPL > 1) {
                v.x = second ? a[1][i] : v.x;
                v.y = second ? a[1][i + 1] : v.y;
            }
            if constexpr (CPL > 2) {
                v.x = third ? a[2][i] : v.x;
                v.y = third ? a[2][i + 1] : v.y;
            }
            *reinterpret_cast<typename Pair<R>::type*>(us + i) = v;
        }
    }
    __syncwarp();
}

// Adds the slabs' values of every column: one barrier.
template <typename R, int NW, int CPL>
__device__ __forceinline__ void sum_slabs(const Cta<R, NW>& C, int buf, R (&s)[CPL]) {
    R* p = C.part(buf);
#pragma unroll
    for (int c = 0; c < CPL; ++c) p[C.warp * C.L.cp + C.lane + 32 * c] = s[c];
    __syncthreads();
#pragma unroll
    for (int c = 0; c < CPL; ++c) {
        R t = R(0);
#pragma unroll
        for (int w = 0; w < NW; ++w) t += p[w * C.L.cp + C.lane + 32 * c];
        s[c] = t;
    }
}

// One elimination step: the reflector of column p on row j (the first row of
// the owning warp's slab), applied to all columns.  On return t holds row j of
// R for this lane's columns, the owner's slab has moved up by one row and us
// holds the warp's part of the reflector's vector u without its entry u0 at
// row j; H = I - tau u u^T. 
template <typename R>
struct Reflector {
    R u0, tau;
};
template <typename R, int NW, int CPL, int RPW>
__device__ __forceinline__ Reflector<R> eliminate(const Cta<R, NW> C, R (&a)[CPL][RPW], int j, int p,
                                                  R* us, R (&t)[CPL]) {
    const int lane = C.lane, buf = j & 1, owner = j / RPW;
    R s[CPL], sigma, alpha;
    if (C.warp == owner) {
#pragma unroll
        for (int c = 0; c < CPL; ++c) {
            C.rowt(buf)[lane + 32 * c] = a[c][0];
            a[c][0] = R(0);
        }
    }
    const bool live = C.warp >= owner;   // the slabs above are finished
#pragma unroll
    for (int c = 0; c < CPL; ++c) s[c] = R(0);
    if (live) {
        publish_column<R, CPL, RPW>(a, p, us, lane);
        slab_dots<R, CPL, RPW>(us, a, s);
    }
    R* q = C.part(buf);
#pragma unroll
    for (int c = 0; c < CPL; ++c) q[C.warp * C.L.cp + lane + 32 * c] = s[c];
    __syncthreads();
    sigma = R(0);
#pragma unroll
    for (int w = 0; w < NW; ++w) sigma += q[w * C.L.cp + p];
    alpha = C.rowt(buf)[p];
#pragma unroll
    for (int c = 0; c < CPL; ++c) {
        t[c] = C.rowt(buf)[lane + 32 * c];
        s[c] = R(0);
#pragma unroll
        for (int w = 0; w < NW; ++w) s[c] += q[w * C.L.cp + lane + 32 * c];
    }
    Reflector<R> H{R(0), R(0)};
    R scal = R(0), tau1 = R(0);   // u / u0 and its factor: safe for columns near underflow
    if (sigma > R(0)) {
        // beta = -sign(alpha) h, h = ||x||; u0 = alpha - beta; tau1 = -u0 / beta
        const R h2 = r_fma(alpha, alpha, sigma), rs = r_rsqrt(h2), h = h2 * rs;
        H.u0 = alpha + r_copysign(h, alpha);
        tau1 = r_fma(r_abs(alpha), rs, R(1));
        scal = reciprocal(H.u0);
        H.tau = tau1 * scal * scal;
    }
#pragma unroll
    for (int c = 0; c < CPL; ++c) {
        const R w = tau1 * r_fma(s[c], scal, t[c]);
        t[c] -= w;
        s[c] = -w * scal;
    }
    if (C.warp == owner) slab_axpy_up<R, CPL, RPW>(us, a, s);
    else if (live) slab_axpy<R, CPL, RPW>(us, a, s);
    return H;
}

// R factor of an m x n matrix held in slabs (QR without pivoting): row j to
// mat[j * ld + c], c < n, for j < min(m, n).
template <typename R, int NW, int CPL, int RPW>
__device__ __forceinline__ void qr_rows(const Cta<R, NW> C, R (&a)[CPL][RPW], int m, int n) {
    const int kk = min(m, n);
    R* mat = C.mat();
    for (int j = 0; j < kk; ++j) {
        R t[CPL];
        eliminate<R, NW, CPL, RPW>(C, a, j, j, C.us(j & 1), t);
        if (C.warp == 0)
#pragma unroll
            for (int c = 0; c < CPL; ++c)
                if (C.lane + 32 * c < n) mat[j * C.L.ld + C.lane + 32 * c] = t[c];
    }
}

// Step 1: R_v of the V stack into mat (min(n, k) rows).
template <typename R, int NW, int CPL, int RPW>
__device__ __noinline__ void phase_rv(const Cta<R, NW> C, const Stack& V) {
    R a[CPL][RPW];
    const int k = V.cols(), row0 = C.warp * RPW;
#pragma unroll
    for (int s = 0; s < CPL; ++s) {
        const int c = C.lane + 32 * s;
        load_slab<R, RPW>(a[s], c < k ? V.col(c) : nullptr, c < k ? V.scale(c) : 0.0, row0, V.rows,
                          c < k);
    }
    qr_rows<R, NW, CPL, RPW>(C, a, V.rows, k);
    __syncthreads();
}

// Steps 2 and 3: T (rows x n) and its pivoted QR.  kind: ROUND_GENERAL (T =
// U R_v^T, R_v's rows in mat), ROUND_ORTHO (T = U), ROUND_DENSE (T = alpha D +
// beta U2 V2^T).  R_1 goes to mat, the reflectors' vectors (zero above their
// row) to refl (column j at refl + j rows), their factors to tau.  Returns k';
// -1 when T holds NaN or Inf.
template <typename R, int NW, int CPL, int RPW>
__device__ __noinline__ int phase_qr(const Cta<R, NW> C, const RoundOp& op, const Stack& U, int n,
                                     R* refl, R tiny_rel, R* tiny_out, int* exponent) {
    const int lane = C.lane, warp = C.warp, rows = U.rows, row0 = warp * RPW;
    R* mat = C.mat();
    R a[CPL][RPW];
    if (op.kind == ROUND_GENERAL) {
#pragma unroll
        for (int s = 0; s < CPL; ++s)
#pragma unroll
            for (int i = 0; i < RPW; ++i) a[s][i] = R(0);
        const int k = U.cols();
        Fetch<R, RPW> f;
        f.get(U.col(0), U.scale(0), row0, rows, lane);
        for (int p = 0; p < k; ++p) {
            R* us = C.us(p & 1);
            f.put(us, lane);
            if (p + 1 < k) f.get(U.col(p + 1), U.scale(p + 1), row0, rows, lane);
            R w[CPL];
#pragma unroll
            for (int s = 0; s < CPL; ++s) {
                const int c = lane + 32 * s;
                w[s] = c < n && p >= c ? mat[c * C.L.ld + p] : R(0);
            }
            slab_axpy<R, CPL, RPW>(us, a, w);
        }
        __syncthreads();   // mat is rewritten below
    } else {
#pragma unroll
        for (int s = 0; s < CPL; ++s) {
            const int c = lane + 32 * s;
            load_slab<R, RPW>(a[s], op.kind == ROUND_DENSE ? op.u1 + (long long)c * op.ldu1
                                                          : U.p1 + (long long)c * U.ld1,
                              op.kind == ROUND_DENSE ? op.alpha : U.s1, row0, rows, c < n);
        }
        if (op.kind == ROUND_DENSE && op.beta != 0.0 && sizeof(R) == 8) {
            for (int l = 0; l < op.r2; ++l) {
                Fetch<R, RPW> f;
                f.get(op.u2 + (long long)l * op.ldu2, op.beta, row0, rows, lane);
                f.put(C.us(l & 1), lane);
                R w[CPL];
#pragma unroll
                for (int s = 0; s < CPL; ++s) {
                    const int c = lane + 32 * s;
                    w[s] = c < n ? (R)op.v2[c + (long long)l * op.ldv2] : R(0);
                }
                slab_axpy<R, CPL, RPW>(C.us(l & 1), a, w);
            }
            __syncwarp();
        } else if (op.kind == ROUND_DENSE && op.beta != 0.0) {
            // FP32: the two parts may cancel, so their sum is taken in FP64, some
            // rows at a time; kept behind the reflectors (work holds rows x n
            // doubles) for V_out
            R* sum = refl + (long long)rows * n;
            constexpr int CH = RPW % 8 == 0 ? 8 : 4;
#pragma unroll
            for (int i0 = 0; i0 < RPW; i0 += CH) {
                double t[CPL][CH], v[CPL], u = 0.0;
                const double* v2[CPL];
                const bool fetches = lane < CH && row0 + i0 + lane < rows;
                const double* u2 = op.u2 + row0 + i0 + lane;
#pragma unroll
                for (int s = 0; s < CPL; ++s) {
                    const int c = min(lane + 32 * s, n - 1);
                    v2[s] = op.v2 + c;
                    v[s] = op.r2 > 0 ? *v2[s] : 0.0;
#pragma unroll
                    for (int q = 0; q < CH; ++q) {
                        const int row = row0 + i0 + q;
                        t[s][q] = row < rows ? op.alpha * op.u1[row + (long long)c * op.ldu1] : 0.0;
                    }
                }
                if (fetches && op.r2 > 0) u = *u2;
                for (int l = 0; l < op.r2; ++l) {
                    double* us = reinterpret_cast<double*>(C.us(l & 1));
                    if (lane < CH) us[lane] = u;
                    __syncwarp();
                    double w[CPL];
#pragma unroll
                    for (int s = 0; s < CPL; ++s) w[s] = op.beta * v[s];
                    if (l + 1 < op.r2) {   // the next column of U2 and V2
                        u2 += op.ldu2;
                        if (fetches) u = *u2;
#pragma unroll
                        for (int s = 0; s < CPL; ++s) {
                            v2[s] += op.ldv2;
                            v[s] = *v2[s];
                        }
                    }
#pragma unroll
                    for (int q = 0; q < CH; q += 2) {
                        const double2 x = *reinterpret_cast<const double2*>(us + q);
#pragma unroll
                        for (int s = 0; s < CPL; ++s) {
                            t[s][q] = fma(x.x, w[s], t[s][q]);
                            t[s][q + 1] = fma(x.y, w[s], t[s][q + 1]);
                        }
                    }
                }
                __syncwarp();
#pragma unroll
                for (int s = 0; s < CPL; ++s)
#pragma unroll
                    for (int q = 0; q < CH; ++q) {
                        const int c = lane + 32 * s, row = row0 + i0 + q;
                        a[s][i0 + q] = c < n && row < rows ? (R)t[s][q] : R(0);
                        if (c < n && row < rows) sum[row + (long long)c * rows] = (R)t[s][q];
                    }
            }
        }
    }
    // T is scaled by a power of two so that its largest entry lies in [1, 2):
    // U_out and the relative thresholds do not depend on the scale
    {
        R mx = R(0);
#pragma unroll
        for (int s = 0; s < CPL; ++s)
#pragma unroll
            for (int i = 0; i < RPW; ++i) mx = r_max(mx, r_abs(a[s][i]));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = r_max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        if (lane == 0) C.part(0)[warp] = mx;
        __syncthreads();
        for (int w = 0; w < NW; ++w) mx = r_max(mx, C.part(0)[w]);
        __syncthreads();
        int e = 0;
        if (mx > R(0) && isfinite((double)mx)) e = ilogb(mx);
        *exponent = e;
        // 2^-e in two factors, each of them representable
        const R f0 = (R)scalbn(1.0, -(e / 2)), f1 = (R)scalbn(1.0, -(e - e / 2));
#pragma unroll
        for (int s = 0; s < CPL; ++s)
#pragma unroll
            for (int i = 0; i < RPW; ++i) a[s][i] = a[s][i] * f0 * f1;
    }
    // squared norms of the columns' remaining parts, the same in every warp
    R nrm[CPL], ref[CPL];
    auto column_norms = [&](int buf) {
#pragma unroll
        for (int s = 0; s < CPL; ++s) {
            R t0 = R(0), t1 = R(0);
#pragma unroll
            for (int i = 0; i < RPW; i += 2) {
                t0 = r_fma(a[s][i], a[s][i], t0);
                t1 = r_fma(a[s][i + 1], a[s][i + 1], t1);
            }
            ref[s] = t0 + t1;
        }
        sum_slabs<R, NW, CPL>(C, buf, ref);
    };
    column_norms(2);
    R fro = R(0);
    unsigned done = 0;   // bit s: this lane's column of slot s is used up
#pragma unroll
    for (int s = 0; s < CPL; ++s) {
        nrm[s] = ref[s];
        fro += ref[s];
        if (lane + 32 * s >= n) done |= 1u << s;
    }
    fro = warp_sum(fro);
    *tiny_out = tiny_rel * fro;
    if (!isfinite((double)fro)) return -1;
    const R tiny = tiny_rel * fro;
    const int kk = min(rows, n);
    int j = 0;
    for (; j < kk; ++j) {
        // pivot: the largest remaining column to 16 bits of its norm (one
        // integer reduction), the lowest index among equals
        unsigned key = 0;
#pragma unroll
        for (int s = 0; s < CPL; ++s)
            if (!((done >> s) & 1) && nrm[s] > R(0))
                key = max(key, (__float_as_uint((float)nrm[s]) & ~0x7fu) | (unsigned)(127 - (lane + 32 * s)));
        key = __reduce_max_sync(0xffffffffu, key);
        const int p = 127 - (int)(key & 0x7fu);
        const R best = (R)__uint_as_float(key & ~0x7fu);
        if (!(best > tiny)) break;   // (key 0: no column left)
        R t[CPL];
        R* us = C.us(j & 1);
        const Reflector<R> H = eliminate<R, NW, CPL, RPW>(C, a, j, p, us, t);
        // the reflector's vector and its row of R_1
        {
            const int owner = j / RPW, first = warp == owner ? j : row0;
            for (int i = lane; i < RPW; i += 32) {
                const int row = first + i;
                if (warp < owner) {
                    if (row < rows) refl[(long long)j * rows + row] = R(0);
                } else if (row < row0 + RPW && row < rows) {
                    refl[(long long)j * rows + row] = row == j ? H.u0 : us[i];
                }
            }
            if (warp == owner)   // zeros above row j in the owner's slab
                for (int row = row0 + lane; row < j; row += 32) refl[(long long)j * rows + row] = R(0);
        }
        if (warp == 0) {
            if (lane == 0) C.tau()[j] = H.tau;
#pragma unroll
            for (int c = 0; c < CPL; ++c)
                if (lane + 32 * c < n) mat[j * C.L.ld + lane + 32 * c] = t[c];
        }
        // norms without the row just finished; formed anew where the
        // subtraction has cancelled too much of them
        bool stale = false;
#pragma unroll
        for (int c = 0; c < CPL; ++c) {
            if (p == lane + 32 * c) done |= 1u << c;
            nrm[c] = r_fma(-t[c], t[c], nrm[c]);
            if (!((done >> c) & 1) && ref[c] > tiny && nrm[c] < R(1e-5) * ref[c]) stale = true;
        }
        if (__any_sync(0xffffffffu, stale)) {
            column_norms(2);
#pragma unroll
            for (int c = 0; c < CPL; ++c) nrm[c] = ref[c];
        }
    }
    __syncthreads();
    return j;
}

// Step 4: R_2 of R_1^T; R_1 (k1 rows of n) is in mat, R_2 (k1 rows) replaces it.
template <typename R, int NW, int CPL, int RPW>
__device__ __noinline__ void phase_lq(const Cta<R, NW> C, int k1, int n) {
    R a[CPL][RPW];
    const int row0 = C.warp * RPW;
    const R* mat = C.mat();
#pragma unroll
    for (int s = 0; s < CPL; ++s) {
        const int c = C.lane + 32 * s;
#pragma unroll
        for (int i = 0; i < RPW; ++i)
            a[s][i] = c < k1 && row0 + i < n ? mat[c * C.L.ld + row0 + i] : R(0);
    }
    __syncthreads();
    qr_rows<R, NW, CPL, RPW>(C, a, n, k1);
    __syncthreads();
}

// Whether two of the n columns (rows of mat, each of `len` entries) are still
// coupled above the threshold; squared norms to nrm.  The Gram matrix in 8 x 8
// tiles on the FP64 tensor pipe, its diagonal first.
template <typename R, int NW>
__device__ __forceinline__ bool coupled(const Cta<R, NW> C, int n, int len, R tiny, R jt2) {
    const R* mat = C.mat();
    R* nrm = C.nrm();
    const int g = C.lane >> 2, t = C.lane & 3, ld = C.L.ld, nt = (n + 7) >> 3;
    auto tile = [&](int ti, int tj, double (&d)[2]) {
        d[0] = d[1] = 0.0;
        const R* pa = mat + min(8 * ti + g, n - 1) * ld;
        const R* pb = mat + min(8 * tj + g, n - 1) * ld;
        double e[2] = {0.0, 0.0};
        for (int k = 0; k < len; k += 8) {
            const double a0 = k + t < len ? (double)pa[k + t] : 0.0;
            const double b0 = k + t < len ? (double)pb[k + t] : 0.0;
            const double a1 = k + 4 + t < len ? (double)pa[k + 4 + t] : 0.0;
            const double b1 = k + 4 + t < len ? (double)pb[k + 4 + t] : 0.0;
            dmma(d, a0, b0);
            dmma(e, a1, b1);
        }
        d[0] += e[0];
        d[1] += e[1];
    };
    if (C.warp == 0 && C.lane == 0) *C.flag() = 0;
    for (int ti = C.warp; ti < nt; ti += NW) {
        double d[2];
        tile(ti, ti, d);
#pragma unroll
        for (int h = 0; h < 2; ++h)
            if (g == 2 * t + h && 8 * ti + g < n) nrm[8 * ti + g] = (R)d[h];
    }
    __syncthreads();
    bool rotate = false;
    for (int q = C.warp; q < nt * (nt + 1) / 2; q += NW) {
        int ti = 0, r = q;
        while (r >= nt - ti) {
            r -= nt - ti;
            ++ti;
        }
        const int tj = ti + r;
        double d[2];
        tile(ti, tj, d);
        const int p = 8 * ti + g;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int c = 8 * tj + 2 * t + h;
            if (p < c && c < n) {
                const R x = (R)d[h], a = nrm[p], b = nrm[c];
                rotate = rotate || (x != R(0) && a > tiny && b > tiny && x * x > jt2 * (a * b));
            }
        }
    }
    if (rotate) *C.flag() = 1;
    __syncthreads();
    const bool again = *C.flag() != 0;
    __syncthreads();
    return again;
}

// The rotation that makes two columns of squared norms a, b and inner product
// c orthogonal, by the smaller angle: with h = sqrt(d^2 + 4 c^2), d = b - a,
// cos^2 = (1 + |d| / h) / 2 and sin cos = |c| / h; t c (t the tangent) is what
// the squared norms change by.
template <typename R>
__device__ __forceinline__ void rotation(R a, R b, R c, R& cs, R& sn, R& tc) {
    const R d = b - a, q = r_fma(d, d, R(4) * c * c), rh = r_rsqrt(q);
    const R x = r_fma(R(0.5) * r_abs(d), rh, R(0.5)), rx = r_rsqrt(x);
    cs = x * rx;
    const R m = r_abs(c) * rh * rx;
    sn = r_copysign(m, d * c);
    tc = r_copysign(r_abs(c) * m * rx, d);
}

// One sweep of one-sided Jacobi over n (even, <= 2 P) columns in odd-even
// order: a lane holds the columns of two neighbouring positions (its share RL
// of their rows), rotates them in registers and interchanges them, so that
// after n steps every pair has met once; between steps one column moves to
// the neighbouring lane.  P lanes hold the pairs, the 32 / P lane groups and
// the NWJ warps hold the row shares.
template <typename R, int NW, int P, int RL, int NWJ>
__device__ __noinline__ void jacobi_sweep(const Cta<R, NW> C, int n, int len, R tiny, R jt2) {
    constexpr int HS = 32 / P;
    const int lane = C.lane, i0 = lane % P, grp = lane / P, np = n >> 1;
    const int r0 = (C.warp * HS + grp) * RL;
    R* mat = C.mat();
    const int ld = C.L.ld;
    R x[RL], y[RL];
    R nx = R(0), ny = R(0);
    const bool on = i0 < np;
#pragma unroll
    for (int i = 0; i < RL; ++i) {
        const bool v = on && r0 + i < len;
        x[i] = v ? mat[(2 * i0) * ld + r0 + i] : R(0);
        y[i] = v ? mat[(2 * i0 + 1) * ld + r0 + i] : R(0);
    }
    if (on) {
        nx = C.nrm()[2 * i0];
        ny = C.nrm()[2 * i0 + 1];
    }
    const int up = grp * P + (on ? (i0 + 1 == np ? 0 : i0 + 1) : i0);
    const int down = grp * P + (on ? (i0 == 0 ? np - 1 : i0 - 1) : i0);
    // rotates (p, q) and interchanges them: p' = sn p + cs q, q' = cs p - sn q
    auto step = [&](bool live, int buf) {
        constexpr int NA = RL < 4 ? RL : 4;
        R cp[NA];
#pragma unroll
        for (int i = 0; i < NA; ++i) cp[i] = x[i] * y[i];
#pragma unroll
        for (int i = NA; i < RL; ++i) cp[i % NA] = r_fma(x[i], y[i], cp[i % NA]);
        R c = NA == 4 ? (cp[0] + cp[1]) + (cp[2] + cp[3]) : cp[0] + cp[1];
#pragma unroll
        for (int o = P; o < 32; o <<= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
        if (NWJ > 1) {
            R* ex = C.jex(buf);
            ex[C.warp * 32 + lane] = c;
            __syncthreads();
            c = R(0);
#pragma unroll
            for (int w = 0; w < NWJ; ++w) c += ex[w * 32 + lane];
        }
        R cs = R(1), sn = R(0), tc = R(0);
        if (c != R(0) && nx > tiny && ny > tiny && c * c > jt2 * (nx * ny)) {
            rotation(nx, ny, c, cs, sn, tc);
        }
        if (live) {
            const R a = nx - tc;
            nx = ny + tc;
            ny = a;
#pragma unroll
            for (int i = 0; i < RL; ++i) {
                const R xi = x[i], yi = y[i];
                x[i] = r_fma(sn, xi, cs * yi);
                y[i] = r_fma(cs, xi, -(sn * yi));
            }
        }
    };
    for (int st = 0; st < n; st += 2) {
        step(true, 0);
        // positions (2i + 1, 2i + 2): the upper lane's first column comes down
#pragma unroll
        for (int i = 0; i < RL; ++i) {
            const R t = __shfl_sync(0xffffffffu, x[i], up);
            x[i] = y[i];
            y[i] = t;
        }
        {
            const R t = __shfl_sync(0xffffffffu, nx, up);
            nx = ny;
            ny = t;
        }
        step(i0 + 1 < np, 1);
#pragma unroll
        for (int i = 0; i < RL; ++i) {
            const R t = __shfl_sync(0xffffffffu, y[i], down);
            y[i] = x[i];
            x[i] = t;
        }
        {
            const R t = __shfl_sync(0xffffffffu, ny, down);
            ny = nx;
            nx = t;
        }
    }
#pragma unroll
    for (int i = 0; i < RL; ++i)
        if (on && r0 + i < len) {
            mat[(2 * i0) * ld + r0 + i] = x[i];
            mat[(2 * i0 + 1) * ld + r0 + i] = y[i];
        }
}

// The same sweep from shared memory for 65 to 96 columns: eight lanes a pair,
// twelve rows a lane, read once and rotated in registers.  A warp's four pairs
// are NW apart, which with an odd ld puts their columns on the same banks
// (FP64) or on different ones (FP32); rows are taken in an order that spreads
// the former.
template <typename R, int NW>
__device__ __noinline__ void jacobi_sweep_wide(const Cta<R, NW> C, int n, int len, R tiny, R jt2) {
    constexpr int RL = 12;   // rows of a lane: up to 96 rows
    R* mat = C.mat();
    R* nrm = C.nrm();
    const int ld = C.L.ld, grp = C.lane >> 3, hl = C.lane & 7;
    const int turn = sizeof(R) == 8 ? grp & 1 : NW == 8 ? grp >> 1 : 0;
    for (int st = 0; st < n; ++st) {
        const int np = (n - (st & 1)) >> 1;   // pairs of this step
        for (int kb = 0; kb < np; kb += 4 * NW) {
            const int k = kb + grp * NW + C.warp;
            const bool live = k < np;
            const int p = live ? 2 * k + (st & 1) : 0;
            R* gp = mat + p * ld;
            R* gq = gp + ld;
            R x[RL], y[RL], cp[4] = {R(0), R(0), R(0), R(0)};
#pragma unroll
            for (int i = 0; i < RL; ++i) {
                const int r = hl + 8 * (i ^ turn);
                const bool v = live && r < len;
                x[i] = v ? gp[r] : R(0);
                y[i] = v ? gq[r] : R(0);
                cp[i & 3] = r_fma(x[i], y[i], cp[i & 3]);
            }
            R c = (cp[0] + cp[1]) + (cp[2] + cp[3]);
            const R nx = nrm[p], ny = nrm[p + 1];
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
            R cs = R(1), sn = R(0), tc = R(0);
            if (c != R(0) && nx > tiny && ny > tiny && c * c > jt2 * (nx * ny)) {
                rotation(nx, ny, c, cs, sn, tc);
            }
#pragma unroll
            for (int i = 0; i < RL; ++i) {
                const int r = hl + 8 * (i ^ turn);
                if (live && r < len) {
                    gp[r] = r_fma(sn, x[i], cs * y[i]);
                    gq[r] = r_fma(cs, x[i], -(sn * y[i]));
                }
            }
            if (live && hl == 0) {   // (every lane has read the norms: the sum above)
                nrm[p] = ny + tc;
                nrm[p + 1] = nx - tc;
            }
        }
        __syncthreads();
    }
}

// Step 5: Jacobi on the k1 rows of mat (upper triangular R_2: row c holds
// column c of L).  Leaves n = k1 rounded up to even columns and their squared
// norms; returns n.
template <typename R, int NW>
__device__ __noinline__ int phase_jacobi(const Cta<R, NW> C, int k1, R tiny) {
    R* mat = C.mat();
    const int n = (k1 + 1) & ~1, ld = C.L.ld;
    // zeros left of the diagonal and in the padding column
    for (int c = C.warp; c < n; c += NW)
        for (int i = C.lane; i < k1; i += 32)
            if (i < c || c >= k1) mat[c * ld + i] = R(0);
    __syncthreads();
    // Couplings left: the rounding of an inner product of k1 terms, from 20
    // columns on above the general kernel's 1e-15, at which sweeps rotate noise
    // (36 x 36 points, rank 46, whose blocks have up to 92 columns: product 82 ms
    // against 61).  Median distance from LAPACK's best approximations of 96
    // columns, of the block's norm and times the gap: 2.3e-17, with 1e-15
    // 1.8e-17; the general kernel's 4.1e-17.
    const R eps = sizeof(R) == 8 ? R(2.220446049250313e-16) : R(1e-6);
    const R jt2 = sizeof(R) == 8 ? eps * eps * R(max(k1, 20)) : eps * eps;
    for (int sweep = 0; sweep < kMaxSweeps && coupled<R, NW>(C, n, k1, tiny, jt2); ++sweep) {
        if (n <= 16) {
            if (C.warp == 0) jacobi_sweep<R, NW, 8, 4, 1>(C, n, k1, tiny, jt2);
        } else if (n <= 32) {
            if (C.warp == 0) jacobi_sweep<R, NW, 16, 16, 1>(C, n, k1, tiny, jt2);
        } else if (n <= 64) {
            jacobi_sweep<R, NW, 32, 64 / NW, NW>(C, n, k1, tiny, jt2);
        } else {
            jacobi_sweep_wide<R, NW>(C, n, k1, tiny, jt2);
        }
        __syncthreads();
    }
    // squared norms of the rotated columns
    R* nrm = C.nrm();
    for (int c = C.warp; c < n; c += NW) {
        R t = R(0);
        for (int i = C.lane; i < k1; i += 32) t = r_fma(mat[c * ld + i], mat[c * ld + i], t);
        t = warp_sum(t);
        if (C.lane == 0) nrm[c] = t;
    }
    __syncthreads();
    return n;
}

// Step 6, first half: U_out = Q_t Y (keep columns, zeros up to rout) to uo,
// and G = U_s^T U_out (k x rout) to mat, or for a dense block V_out itself.
template <typename R, int NW, int CPL, int RPW>
__device__ __noinline__ void phase_u(const Cta<R, NW> C, const RoundOp& op, const Stack& U, int n,
                                     const R* refl, int k1, int keep, R tiny, double* uo,
                                     double* vo) {
    const int lane = C.lane, warp = C.warp, rows = U.rows, row0 = warp * RPW, rout = op.rout;
    const int ld = C.L.ld, rp = C.L.rp;
    R* mat = C.mat();
    R a[CPL][RPW];
#pragma unroll
    for (int s = 0; s < CPL; ++s) {
        const int c = lane + 32 * s;
        int src = 0;
        R inv = R(0);
        if (c < keep) {
            src = C.order()[c];
            const R q = C.nrm()[src];
            if (q > tiny) inv = R(1) / r_sqrt(q);   // noise columns are dropped
        }
#pragma unroll
        for (int i = 0; i < RPW; ++i)
            a[s][i] = inv != R(0) && row0 + i < k1 ? inv * mat[src * ld + row0 + i] : R(0);
    }
    {
        const R* col = refl + (long long)(k1 - 1) * rows;
        R v0 = R(0), v1 = R(0);
        auto get = [&]() {
            v0 = lane < RPW && row0 + lane < rows ? col[row0 + lane] : R(0);
            if (RPW > 32) v1 = 32 + lane < RPW && row0 + 32 + lane < rows ? col[row0 + 32 + lane] : R(0);
        };
        get();
        for (int j = k1 - 1; j >= 0; --j) {
            const int buf = j & 1;
            R* us = C.us(buf);
            if (lane < RPW) us[lane] = v0;
            if (RPW > 32 && 32 + lane < RPW) us[32 + lane] = v1;
            __syncwarp();
            col -= rows;
            if (j > 0) get();
            R s[CPL];
            slab_dots<R, CPL, RPW>(us, a, s);
            sum_slabs<R, NW, CPL>(C, buf, s);
            const R t = -C.tau()[j];
#pragma unroll
            for (int c = 0; c < CPL; ++c) s[c] *= t;
            slab_axpy<R, CPL, RPW>(us, a, s);
        }
    }
#pragma unroll
    for (int s = 0; s < CPL; ++s) {
        const int c = lane + 32 * s;
        if (c < rout)
#pragma unroll
            for (int i = 0; i < RPW; ++i)
                if (row0 + i < rows) uo[row0 + i + (long long)c * rows] = (double)a[s][i];
    }
    __syncthreads();   // mat and the buffers are rewritten
    // inner products of `count` columns with U_out, kChunk per barrier;
    // fetch(p, f) brings column p, finish(p, c, value) runs once per product
    auto products = [&](int count, auto fetch, auto finish) {
        Fetch<R, RPW> f;
        if (count > 0) fetch(0, f);
        for (int p0 = 0; p0 < count; p0 += kChunk) {
            const int buf = (p0 / kChunk) & 1, nc = min(kChunk, count - p0);
            R* ch = C.chunk(buf);
            for (int q = 0; q < nc; ++q) {
                R* us = C.us(q & 1);
                f.put(us, lane);
                if (p0 + q + 1 < count) fetch(p0 + q + 1, f);
                R s[CPL];
                slab_dots<R, CPL, RPW>(us, a, s);
#pragma unroll
                for (int c = 0; c < CPL; ++c)
                    if (lane + 32 * c < rp) ch[(warp * kChunk + q) * rp + lane + 32 * c] = s[c];
            }
            __syncthreads();
            for (int q = warp; q < nc; q += NW)
                for (int c = lane; c < rout; c += 32) {
                    R t = R(0);
                    for (int w = 0; w < NW; ++w) t += ch[(w * kChunk + q) * rp + c];
                    finish(p0 + q, c, t);
                }
        }
        __syncthreads();
    };
    if (op.kind != ROUND_DENSE) {
        products(U.cols(), [&](int p, Fetch<R, RPW>& f) { f.get(U.col(p), U.scale(p), row0, rows, lane); },
                 [&](int p, int c, R t) { mat[p * ld + c] = t; });
        return;
    }
    const int r2 = op.beta != 0.0 ? op.r2 : 0;
    if (sizeof(R) == 4 && r2 > 0) {
        const R* sum = refl + (long long)rows * n;   // alpha D + beta U2 V2^T (phase_qr)
        products(n,
                 [&](int p, Fetch<R, RPW>& f) {
                     const R* col = sum + (long long)p * rows + row0;
                     f.v0 = lane < RPW && row0 + lane < rows ? col[lane] : R(0);
                     if (RPW > 32) f.v1 = 32 + lane < RPW && row0 + 32 + lane < rows ? col[32 + lane] : R(0);
                 },
                 [&](int p, int c, R t) { vo[p + (long long)c * n] = (double)t; });
        return;
    }
    products(r2, [&](int p, Fetch<R, RPW>& f) { f.get(op.u2 + (long long)p * op.ldu2, op.beta, row0, rows, lane); },
             [&](int p, int c, R t) { mat[p * ld + c] = t; });
    products(n, [&](int p, Fetch<R, RPW>& f) { f.get(op.u1 + (long long)p * op.ldu1, op.alpha, row0, rows, lane); },
             [&](int p, int c, R t) {
                 for (int l = 0; l < r2; ++l) t = r_fma((R)op.v2[p + (long long)l * op.ldv2], mat[l * ld + c], t);
                 vo[p + (long long)c * n] = (double)t;
             });
}

// Step 6, second half: V_out = V_s G.
template <typename R, int NW, int CPL, int RPW>
__device__ __noinline__ void phase_v(const Cta<R, NW> C, const Stack& V, int rout, double* vo) {
    const int lane = C.lane, rows = V.rows, row0 = C.warp * RPW, k = V.cols(), ld = C.L.ld;
    const R* mat = C.mat();
    R a[CPL][RPW];
#pragma unroll
    for (int s = 0; s < CPL; ++s)
#pragma unroll
        for (int i = 0; i < RPW; ++i) a[s][i] = R(0);
    Fetch<R, RPW> f;
    f.get(V.col(0), V.scale(0), row0, rows, lane);
    for (int p = 0; p < k; ++p) {
        R* us = C.us(p & 1);
        f.put(us, lane);
        if (p + 1 < k) f.get(V.col(p + 1), V.scale(p + 1), row0, rows, lane);
        R w[CPL];
#pragma unroll
        for (int s = 0; s < CPL; ++s) {
            const int c = lane + 32 * s;
            w[s] = c < rout ? mat[p * ld + c] : R(0);
        }
        slab_axpy<R, CPL, RPW>(us, a, w);
    }
#pragma unroll
    for (int s = 0; s < CPL; ++s) {
        const int c = lane + 32 * s;
        if (c < rout)
#pragma unroll
            for (int i = 0; i < RPW; ++i)
                if (row0 + i < rows) vo[row0 + i + (long long)c * rows] = (double)a[s][i];
    }
}

// Calls CALL(columns per lane, slab rows) for the smallest slab that holds
// `rows` rows in nw warps with `cols` columns.
#define HMB_SLABS(cols, rows, nw, CALL)                                       \
    do {                                                                      \
        const int need_ = ((rows) + (nw) - 1) / (nw);                         \
        constexpr bool wide_ = sizeof(R) == 4;   /* FP32: twice the rows */   \
        if ((cols) <= 32) {                                                   \
            if (need_ <= 8) { CALL(1, 8); }                                   \
            else if (need_ <= 16) { CALL(1, 16); }                            \
            else if (need_ <= 24) { CALL(1, 24); }                            \
            else if (!wide_ || need_ <= 32) { CALL(1, 32); }                  \
            else { CALL(1, (wide_ ? 64 : 32)); }                              \
        } else if ((cols) <= 64) {                                            \
            if (need_ <= 8) { CALL(2, 8); }                                   \
            else if (!wide_ || need_ <= 16) { CALL(2, 16); }                  \
            else { CALL(2, (wide_ ? 32 : 16)); }                              \
        } else {                                                              \
            if (!wide_ || need_ <= 12) { CALL(3, 12); }                       \
            else { CALL(3, (wide_ ? 24 : 12)); }                              \
        }                                                                     \
    } while (0)

// One GENERAL, DENSE or ORTHO rounding by the whole CTA.
template <typename R, int NW>
__device__ void round_in_registers(const RoundOp& op, const Cta<R, NW> C, R tiny_rel, double tol_floor,
                                   int* numflag) {
    const int tid = C.warp * 32 + C.lane;
    const bool dense = op.kind == ROUND_DENSE, ortho = op.kind == ROUND_ORTHO;
    const int m = op.m, n = op.n, rout = op.rout;
    if (m == 0 || n == 0) return;
    Stack U, V;
    double* uo = op.uo;
    double* vo = op.vo;
    if (ortho) {   // (Q_1 Z^T)^T = Z Q_1^T
        U = {op.v1, nullptr, 1.0, 0.0, n, op.r1, 0, op.ldv1, 0};
        V = {op.u1, nullptr, 1.0, 0.0, m, op.r1, 0, op.ldu1, 0};
        uo = op.vo;
        vo = op.uo;
    } else {
        const int r1 = dense ? 0 : op.r1, r2 = op.r2;
        U = {op.u1, op.u2, op.alpha, op.beta, m, r1, r2, op.ldu1, op.ldu2};
        V = {op.v1, op.v2, 1.0, 1.0, n, r1, r2, op.ldv1, op.ldv2};
    }
    const int k = dense ? n : U.cols();
    const int ku = ortho ? op.r1 : min(m, k), kv = dense ? n : min(n, k);
    const int nt = dense ? n : ortho ? k : kv;   // columns of T
    R* refl = reinterpret_cast<R*>(op.work);
    int k1 = 0, exponent = 0;
    R tiny = R(0);
    if (k > 0) {
        if (op.kind == ROUND_GENERAL) {
#define CALL(c, r) phase_rv<R, NW, c, r>(C, V)
            HMB_SLABS(k, V.rows, NW, CALL);
#undef CALL
        }
#define CALL(c, r) k1 = phase_qr<R, NW, c, r>(C, op, U, nt, refl, tiny_rel, &tiny, &exponent)
        HMB_SLABS(nt, U.rows, NW, CALL);
#undef CALL
    }
    int keep = min(rout, min(ku, kv));
    if (k1 <= 0) {
        // zero, or not finite: the rank the tolerance rule gives a zero block
        const double fill = k1 < 0 ? (double)NAN : 0.0;
        if (k1 < 0 && tid == 0 && numflag) atomicOr(numflag, 1);
        if (op.tol > 0.0 && keep > 0) keep = 1;
        if (tid == 0 && op.rank_out) *op.rank_out = keep;
        for (int c = C.warp; c < rout; c += NW) {
            for (int i = C.lane; i < m; i += 32) op.uo[i + (long long)c * m] = c < keep ? fill : 0.0;
            for (int i = C.lane; i < n; i += 32) op.vo[i + (long long)c * n] = c < keep ? fill : 0.0;
        }
        return;
    }
#define CALL(c, r) phase_lq<R, NW, c, r>(C, k1, nt)
    HMB_SLABS(k1, nt, NW, CALL);
#undef CALL
    const int nc = phase_jacobi<R, NW>(C, k1, tiny);
    // columns by decreasing norm (ties by index)
    const R* nrm = C.nrm();
    for (int j = tid; j < nc; j += NW * 32) {
        const R sj = nrm[j] == nrm[j] ? nrm[j] : R(-1);
        int pos = 0;
        for (int i = 0; i < nc; ++i) {
            const R si = nrm[i] == nrm[i] ? nrm[i] : R(-1);
            pos += (si > sj || (si == sj && i < j)) ? 1 : 0;
        }
        C.order()[pos] = j;
    }
    __syncthreads();
    if (op.tol > 0.0 && keep > 0) {
        // SVDTrunc: sigma_0, and every sigma above tol sigma_0 unless
        // sigma_0 < tol^2
        const double s0 = nrm[C.order()[0]];
        const double tol = op.tol > tol_floor ? op.tol : tol_floor, t2 = tol * tol;
        int c = 1;
        if (scalbn(sqrt(s0), exponent) >= t2)
            while (c < keep && c < nc && (double)nrm[C.order()[c]] > t2 * s0) ++c;
        keep = c;
    }
    if (tid == 0 && op.rank_out) *op.rank_out = keep;
    const int cols = min(keep, nc);
    if (rout > 0) {
#define CALL(c, r) phase_u<R, NW, c, r>(C, op, U, nt, refl, k1, cols, tiny, uo, vo)
        HMB_SLABS(rout, U.rows, NW, CALL);
#undef CALL
        if (ortho && sizeof(R) == 4) {
            // FP32: the orthonormal factor stays as it is, its combinations in FP64
            const R* mat = C.mat();
            for (int c = C.warp; c < rout; c += NW)
                for (int i = C.lane; i < V.rows; i += 32) {
                    double t = 0.0;
                    for (int p = 0; p < k; ++p)
                        t = fma(V.p1[i + (long long)p * V.ld1], (double)mat[p * C.L.ld + c], t);
                    vo[i + (long long)c * V.rows] = t;
                }
        } else if (!dense) {
#define CALL(c, r) phase_v<R, NW, c, r>(C, V, rout, vo)
            HMB_SLABS(rout, V.rows, NW, CALL);
#undef CALL
        }
    }
}

}  // namespace reground
}  // namespace hmb
