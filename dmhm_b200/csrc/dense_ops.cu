// Batched small dense products for the leaf algebra of the H*H product:
// C = alpha op(A) op(B) + beta C, one CTA per product, 64 x 64 output tiles.
//
// These replace the reference's per-leaf BLAS calls in the dense and
// low-rank leaf products (src/hmat_tools/MultiplyMatrix.cpp:31-450: D*D,
// D*F, F*D, F*F, and the dense updates of src/hmat_tools/Update.cpp:14-108),
// which the reference issues one gemm at a time.
#include "dense_ops.h"

#include <algorithm>

#include "fp64_tiles.cuh"
#include "kernel_limits.h"

namespace hmb {

namespace {

constexpr int kT = 128;   // 4 warps of 16 rows x 64 columns
constexpr int kKC = 16;   // inner chunk
constexpr int kStages = 3;
constexpr int kStage = kKC * 66;   // doubles of one operand's stage
constexpr size_t kSmem = 2ull * kStages * kStage * sizeof(double);

__device__ __forceinline__ double ld_op(const double* X, int ld, bool trans, int i, int j) {
    return trans ? X[j + (long long)i * ld] : X[i + (long long)j * ld];
}

// Stages 16 inner indices of one operand: `wide` (at most 64) rows of op(A) or
// columns of op(B) from X, whose inner index runs with stride 1 (inner) or ld.
// Inner-contiguous operands are staged as rows of 16 inner indices, their
// 16-byte units exchanged between halves on odd rows, the others as columns of
// 64 with a stride of 66: copies and fragment loads then touch each bank once.
__device__ __forceinline__ void stage_operand(unsigned d, const double* X, int ld, bool inner, int wide,
                                              int len, const double* any) {
    const int tid = threadIdx.x;
    const bool al = ((reinterpret_cast<size_t>(X) | (size_t)((long long)ld << 3)) & 15) == 0;
    if (inner) {
        const int u = tid & 7, r0 = tid >> 3;
        const int bytes = max(0, min(16, (len - 2 * u) * 8));
        const double* src = X + 2 * u + (long long)r0 * ld;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int r = r0 + 16 * q;
            if (16 * q < ((wide + 7) & ~7))   // (whole blocks of 8 are multiplied)
                copy_pair(d + (unsigned)(r * kKC + 2 * (u ^ ((r & 1) << 2))) * 8, src,
                          r < wide ? bytes : 0, al, any);
            src += 16LL * ld;
        }
    } else {
        const int u = tid & 31, p0 = tid >> 5;
        const int bytes = max(0, min(16, (wide - 2 * u) * 8));
        const double* src = X + 2 * u + (long long)p0 * ld;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int p = p0 + 4 * q;
            copy_pair(d + (unsigned)(p * 66 + 2 * u) * 8, src, p < len ? bytes : 0, al, any);
            src += 4LL * ld;
        }
    }
}

// Fragment of 8 rows (columns) b .. b + 7 of a staged operand for the inner
// indices 8 kp + 2 t (x) and 8 kp + 2 t + 1 (y).
__device__ __forceinline__ double2 fragment(const double* S, bool inner, int b, int kp, int g, int t) {
    if (inner)
        return *reinterpret_cast<const double2*>(S + (b + g) * kKC + 2 * ((((g & 1) << 2) ^ t) ^ (4 * kp)));
    const double* p = S + (8 * kp + 2 * t) * 66 + b + g;
    return make_double2(p[0], p[66]);
}

__device__ __forceinline__ GemmOp resolve(const GemmOp& src, const RelocBases& bases) {
    GemmOp op = src;
    op.A = reloc(op.A, bases);
    op.B = reloc(op.B, bases);
    op.C = reloc(op.C, bases);
    return op;
}

// Ops [b0, b1), all on one C of m x n, on its 64 x 64 tile at (i0, j0), in
// order.  The products accumulate in registers: C is read at most once (when
// the first product keeps it) and written once, and the chunks of the next
// product are fetched while this one is multiplied.  k < 0 (C = alpha A +
// beta C, whose A may be C itself) goes through memory in between.
// Bound by the FP64 tensor pipe (64 x 64 x 64 products; narrow ones by
// latency); blocks of 8 columns beyond n and warps beyond m do not multiply.
// Measured, 32^3 A A (125 k leaf updates, 113 k leaf products): 4.8 -> 3.4
// and 4.1 -> 3.5 ms; SchulzInvert 72 x 68 (81-point leaves): 80 -> 40 ms of both.
__device__ void gemm_tile(const GemmOp* ops, int b0, int b1, int i0, int j0, const RelocBases& bases,
                          double* sm) {
    __shared__ int4 meta[kStages];      // op, inner indices, layouts, -
    __shared__ double2 scale[kStages];  // alpha, beta
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    double* const As = sm;
    double* const Bs = sm + kStages * kStage;
    const unsigned as0 = (unsigned)__cvta_generic_to_shared(As);
    const unsigned bs0 = (unsigned)__cvta_generic_to_shared(Bs);
    GemmOp cur = resolve(ops[b0], bases);
    const int m = min(64, cur.m - i0), n = min(64, cur.n - j0), ldc = cur.ldc;
    double* const Cb = cur.C + i0 + (long long)j0 * ldc;
    const int ncnt = (n + 7) >> 3;
    const bool live = 16 * warp < m;
    double acc[2][8][2];
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int c = 0; c < 8; ++c) acc[a][c][0] = acc[a][c][1] = 0.0;
    double keep = 1.0;   // C = keep C + acc

    // ---- loader: op lo, inner offset lp -----------------------------------
    int lo = b0, lp = 0;
    auto settle = [&]() {   // the next op with chunks
        while (lo < b1 && cur.k <= 0) {
            ++lo;
            if (lo < b1) cur = resolve(ops[lo], bases);
        }
    };
    settle();
    auto load = [&](int s) {
        if (lo < b1) {
            const int len = min(kKC, cur.k - lp);
            const bool ai = cur.transA != 0, bi = cur.transB == 0;
            const double* any = reinterpret_cast<const double*>(reinterpret_cast<size_t>(cur.A) & ~(size_t)15);
            const double* A = ai ? cur.A + lp + (long long)i0 * cur.lda : cur.A + i0 + (long long)lp * cur.lda;
            const double* B = bi ? cur.B + lp + (long long)j0 * cur.ldb : cur.B + j0 + (long long)lp * cur.ldb;
            stage_operand(as0 + (unsigned)s * (kStage * 8), A, cur.lda, ai, m, len, any);
            stage_operand(bs0 + (unsigned)s * (kStage * 8), B, cur.ldb, bi, n, len, any);
            if (tid == 0) {
                meta[s] = make_int4(lo, len, (ai ? 1 : 0) | (bi ? 2 : 0) | (lp == 0 ? 4 : 0), 0);
                scale[s] = make_double2(cur.alpha, cur.beta);
            }
            lp += len;
            if (lp >= cur.k) {
                lp = 0;
                ++lo;
                if (lo < b1) cur = resolve(ops[lo], bases);
                settle();
            }
        } else if (tid == 0) {
            meta[s] = make_int4(b1, 0, 0, 0);
        }
        cp_async_commit();
    };

    auto each = [&](auto f) {   // f(element of C, accumulator) over this thread's part of the tile
#pragma unroll
        for (int a = 0; a < 2; ++a) {
            const int i = 16 * warp + 8 * a + g;
            if (i >= m) continue;
#pragma unroll
            for (int c = 0; c < 8; ++c)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int j = 8 * c + 2 * t + h;
                    if (j < n) f(Cb + i + (long long)j * ldc, acc[a][c][h]);
                }
        }
    };
    auto flush = [&]() {
        each([&](double* c, double& v) {
            *c = keep == 0.0 ? v : keep == 1.0 ? *c + v : keep * *c + v;
            v = 0.0;
        });
        keep = 1.0;
    };
    bool pending = false;   // acc or keep hold something C does not
    const int shift = m <= 8 ? 3 : m <= 16 ? 4 : m <= 32 ? 5 : 6;   // rows, as a power of two
    // an op without inner indices, in its turn
    auto plain = [&](int o) {
        const GemmOp op = resolve(ops[o], bases);
        if (pending) flush();
        pending = false;
        __syncthreads();   // C may be read by other threads than wrote it
        const bool read = op.k != 0 && op.alpha != 0.0;
        for (int e0 = tid; e0 < n << shift; e0 += 4 * kT) {
            double a[4], v[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {   // all reads first: C may be A
                const int e = e0 + q * kT, i = e & ((1 << shift) - 1), j = e >> shift;
                const bool ok = i < m && j < n;
                a[q] = ok && read ? op.alpha * ld_op(op.A, op.lda, op.transA, i0 + i, j0 + j) : 0.0;
                v[q] = ok && op.beta != 0.0 ? Cb[i + (long long)j * ldc] : 0.0;
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int e = e0 + q * kT, i = e & ((1 << shift) - 1), j = e >> shift;
                if (i < m && j < n) Cb[i + (long long)j * ldc] = op.beta == 0.0 ? a[q] : a[q] + op.beta * v[q];
            }
        }
        __syncthreads();
    };

    int done = b0, s = 0;
    if (lo >= b1) {   // copies and scalings only
        while (done < b1) plain(done++);
        return;
    }
#pragma unroll
    for (int q = 0; q < kStages - 1; ++q) load(q);
    for (;;) {
        cp_async_wait<kStages - 2>();
        __syncthreads();
        const int4 mt = meta[s];
        if (mt.x >= b1) break;
        const double2 ab = scale[s];
        load(s == 0 ? kStages - 1 : s - 1);
        if (mt.z & 4) {   // a new product: what comes before it, then its beta
            while (done < mt.x) plain(done++);
            ++done;
            if (ab.y != 1.0) {
#pragma unroll
                for (int a = 0; a < 2; ++a)
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        acc[a][c][0] = ab.y == 0.0 ? 0.0 : acc[a][c][0] * ab.y;
                        acc[a][c][1] = ab.y == 0.0 ? 0.0 : acc[a][c][1] * ab.y;
                    }
                keep *= ab.y;
            }
            pending = true;
        }
        const double* A = As + s * kStage;
        const double* B = Bs + s * kStage;
        if (live) {
#pragma unroll
            for (int kp = 0; kp < kKC / 8; ++kp) {
                if (8 * kp >= mt.y) break;
                double2 a0 = fragment(A, mt.z & 1, 16 * warp, kp, g, t);
                double2 a1 = fragment(A, mt.z & 1, 16 * warp + 8, kp, g, t);
                if (ab.x != 1.0) {
                    a0.x *= ab.x;
                    a0.y *= ab.x;
                    a1.x *= ab.x;
                    a1.y *= ab.x;
                }
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    if (c < ncnt) {
                        const double2 b = fragment(B, mt.z & 2, 8 * c, kp, g, t);
                        dmma(acc[0][c], a0.x, b.x);
                        dmma(acc[1][c], a1.x, b.x);
                        dmma(acc[0][c], a0.y, b.y);
                        dmma(acc[1][c], a1.y, b.y);
                    }
                }
            }
        }
        s = s + 1 == kStages ? 0 : s + 1;
    }
    while (done < b1) plain(done++);
    if (pending) flush();
    cp_async_wait<0>();
}

// One CTA per (op, 64x64 output tile).
__global__ void __launch_bounds__(kT, 3)
gemm_ops_kernel(const GemmOp* __restrict__ ops, const int* __restrict__ tile_op,
                const int* __restrict__ tile_id, const RelocBases bases) {
    extern __shared__ __align__(16) double gemm_smem[];
    const int o = tile_op[blockIdx.x], tile = tile_id[blockIdx.x], tm = (ops[o].m + 63) / 64;
    gemm_tile(ops, o, o + 1, (tile % tm) * 64, (tile / tm) * 64, bases, gemm_smem);
}

// One CTA per worker and 64 x 64 tile of its C: ops [begin[w], begin[w+1]) in
// order, all on that C.
__global__ void __launch_bounds__(kT, 3)
gemm_worker_kernel(const GemmOp* __restrict__ ops, const int* __restrict__ begin,
                   const RelocBases bases) {
    extern __shared__ __align__(16) double gemm_smem[];
    const int b0 = begin[blockIdx.x], b1 = begin[blockIdx.x + 1], tile = blockIdx.y;
    if (b0 >= b1) return;
    const int tm = (ops[b0].m + 63) / 64, tn = (ops[b0].n + 63) / 64;
    if (tile < tm * tn) gemm_tile(ops, b0, b1, (tile % tm) * 64, (tile / tm) * 64, bases, gemm_smem);
}

}  // namespace

void upload_gemm_tiles(Context& ctx, const std::vector<GemmOp>& ops, GemmTileList& out) {
    out.ntiles = 0;
    std::vector<int> tile_op, tile_id;
    for (size_t o = 0; o < ops.size(); ++o) {
        const GemmOp& g = ops[o];
        if (g.m <= 0 || g.n <= 0) continue;
        int tiles = ceil_div(g.m, 64) * ceil_div(g.n, 64);
        for (int t = 0; t < tiles; ++t) {
            tile_op.push_back((int)o);
            tile_id.push_back(t);
        }
    }
    if (tile_op.empty()) return;
    out.ops.upload(ops, ctx.stream);
    out.tile_op.upload(tile_op, ctx.stream);
    out.tile_id.upload(tile_id, ctx.stream);
    out.ntiles = (int)tile_op.size();
}

void launch_gemm_tiles(Context& ctx, const GemmTileList& L, const RelocBases& bases,
                       const char* name) {
    if (L.ntiles == 0) return;
    allow_smem(gemm_ops_kernel, kSmem);
    LaunchScope ls(ctx, name);
    gemm_ops_kernel<<<(unsigned)L.ntiles, kT, kSmem, ctx.stream>>>(L.ops.get(), L.tile_op.get(),
                                                               L.tile_id.get(), bases);
    HMB_CHECK_LAUNCH();
}

void launch_gemm_ops(Context& ctx, const std::vector<GemmOp>& ops, const char* name) {
    GemmTileList L;
    upload_gemm_tiles(ctx, ops, L);
    launch_gemm_tiles(ctx, L, RelocBases{}, name);
}

void upload_gemm_list(Context& ctx, const std::vector<GemmOp>& ops, const std::vector<int>& begin,
                      GemmList& out) {
    out.nw = 0;
    if (ops.empty() || begin.size() < 2) return;
    out.ops.upload(ops, ctx.stream);
    out.begin.upload(begin, ctx.stream);
    out.nw = (int)begin.size() - 1;
    out.tiles = 1;
    for (const GemmOp& g : ops) out.tiles = std::max(out.tiles, ceil_div(g.m, 64) * ceil_div(g.n, 64));
}

void launch_gemm_list(Context& ctx, const GemmList& L, const RelocBases& bases, const char* name) {
    if (L.nw == 0) return;
    allow_smem(gemm_worker_kernel, kSmem);
    LaunchScope ls(ctx, name);
    gemm_worker_kernel<<<dim3((unsigned)L.nw, (unsigned)L.tiles), kT, kSmem, ctx.stream>>>(L.ops.get(), L.begin.get(), bases);
    HMB_CHECK_LAUNCH();
}

void launch_gemm_workers(Context& ctx, const std::vector<GemmOp>& ops,
                         const std::vector<int>& begin, const char* name) {
    GemmList L;
    upload_gemm_list(ctx, ops, begin, L);
    launch_gemm_list(ctx, L, RelocBases{}, name);
}

}  // namespace hmb
