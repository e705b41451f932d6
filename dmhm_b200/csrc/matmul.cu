// Level-batched H-matrix x dense products (the H-matvec / H-matmat hot path).
//
// Replaces the reference's recursive HMat2d::Multiply / TransposeMultiply
// (src/HMat2d/MultiplyVector-incl.hpp:12-124, MultiplyDense-incl.hpp:12-150),
// which issues one gemv/gemm per dense leaf (src/hmat_tools/MultiplyVector.cpp
// :14-69) and two per low-rank block (:71-128), recursing over the tree.
//
// A job is one subtree (root block, op) of one H-matrix applied to one dense
// input.  Each (H-matrix, root, op) has a template -- its work lists, built
// once and kept on the device -- and a batch of jobs runs as two launches:
//   phase 1: T_b = W_b^T X_b for every low-rank block b of every job
//            (W = V, or U for the transpose): for one column the blocks' rows
//            shared out evenly among warps; otherwise tiles of 64 columns of
//            the W's that share a source box, in chunks of 16 inner indices
//            shared out evenly among persistent CTAs;
//   phase 2: for every output row tile of every job, Y_tile = alpha * (sum
//            over the dense leaves and low-rank blocks covering the tile of
//            A_e(tile rows) * B_e) + beta * Y_tile, shared out likewise; a
//            tile cut between warps or CTAs is added up in their order by the
//            one that finishes last, so each output element is written once
//            and the sums do not depend on the timing.
// Every stored matrix entry is read exactly once per launch pair.  A CTA finds
// its job by binary search over the jobs' first work-item indices.
#include <algorithm>
#include <tuple>
#include <type_traits>
#include <cstring>
#include <map>

#include "engine.h"
#include "fp64_tiles.cuh"
#include "kernel_limits.h"
#include "templates.h"

namespace hmb {

// What a CTA needs to run its share of one job.
struct JobExec {
    const double* hb;    // storage of the job's H-matrix (work lists hold offsets)
    const float* hb32;   // TF32 path: its TF32-rounded FP32 copy
    const float* in32;   // TF32 path: the input, rounded, ld ldin32
    float* T32;          // TF32 path: phase-1 results
    int ldin32, pad32;
    const P1T* p1;
    const W1Tile* w1;
    const int* w1cp;     // wide: chunk prefix over the W1 tiles (n_w1 + 1)
    const int* tcp;      // wide: chunk prefix over the row tiles (n2 + 1)
    const int* ekc;      // wide: first chunk of each entry within its tile
    const WideChunk* ch1;   // wide: chunks of phase 1 / 2
    const WideChunk* ch2;
    double* part;        // wide: partials of tiles cut between CTAs (shared by all jobs)
    const P2T* p2;
    const P2Entry* ent;
    const double* in;
    double* out;
    double* T;
    int* cnt1;           // per item: pieces finished (zero between launches)
    int* cnt2;           // per row tile: pieces finished
    const double* alpha_scale;
    double alpha, beta;
    long long p1_begin, p2_begin;   // first global work item (row / column) of this job
    int n1, n2, ldin, ldout, k, ct1, ct2, pad;   // ct*: column tiles per item
};

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr size_t kLayoutGroups = 16;   // layout groups kept per context

__device__ __forceinline__ int find_job(const JobExec* jobs, int njobs, long long idx,
                                        bool phase2) {
    int lo = 0, hi = njobs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        const long long b = phase2 ? jobs[mid].p2_begin : jobs[mid].p1_begin;
        if (b <= idx) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// ---------------------------------------------------------------------------
// Phase 1: T = W^T in
// ---------------------------------------------------------------------------
// Sum of v[f] over the 32 lanes for 16 values at once (a transposing
// butterfly: 16 shuffles instead of 80).  Lanes 2f and 2f+1 end up holding
// the total of value f in v[0].
__device__ __forceinline__ void warp_transpose_sum16(double (&v)[16], int lane) {
#pragma unroll
    for (int h = 8, o = 16; h >= 1; h >>= 1, o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < h; ++i) {
            const double send = up ? v[i] : v[i + h];
            const double keep = up ? v[i + h] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// Even split of a concatenation of C work items (rows of the phase-1 items,
// columns of the phase-2 tiles, over all jobs) among GW <= C warps: warp w
// takes [w C / GW, (w+1) C / GW), never empty.  An item or tile cut between
// warps wa..wb is summed by the piece that finishes last (a counter per item
// or tile, reset by that piece), over the warps in order; warp w leaves the
// partial sum of its first piece in scratch slot 2w, of its last in 2w + 1.
__device__ __forceinline__ long long split_start(long long w, long long GW, long long C) {
    return w * C / GW;
}
__device__ __forceinline__ long long split_owner(long long g, long long GW, long long C) {
    return ((g + 1) * GW + C - 1) / C - 1;
}
__device__ __forceinline__ long long piece_slot(long long q, long long wa, bool wa_starts_here) {
    return 2 * q + ((q == wa && !wa_starts_here) ? 1 : 0);
}

// One column.  Persistent warps stream their share of the items' rows.  A
// lane owns rows p and p + 32 of a 64-row step and loads JC = 16 columns of W
// for both (2 JC loads in flight); the 16 partial sums of a column chunk
// are reduced across the warp by a transposing butterfly.
__global__ void __launch_bounds__(kThreads, 2)
p1_stream_kernel(const JobExec* __restrict__ jobs, int njobs, const JobExec job0, long long C,
                 long long GW, double* __restrict__ S, int rmax,
                 const int* __restrict__ start) {
    constexpr int JC = 16;
    const int lane = threadIdx.x & 31;
    const long long w = (long long)blockIdx.x * kWarps + (threadIdx.x >> 5);
    if (w >= GW) return;
    const long long slot_len = rmax;
    long long g = split_start(w, GW, C);
    const long long gend = split_start(w + 1, GW, C);
    bool first = true;
    // one job with precomputed starts: items follow one another
    const bool seq = jobs == nullptr && start != nullptr;
    int item = seq ? start[w] - 1 : 0;
    while (g < gend) {
        const JobExec& J = jobs ? jobs[find_job(jobs, njobs, g, false)] : job0;
        const long long local = g - J.p1_begin;
        if (seq) {
            ++item;
        } else {
            item = 0;
            int hi = J.n1 - 1;
            while (item < hi) {
                const int mid = (item + hi + 1) >> 1;
                if (J.p1[mid].c0 <= local) item = mid;
                else hi = mid - 1;
            }
        }
        const P1T it = J.p1[item];
        if (item + 1 < J.n1) asm volatile("prefetch.global.L1 [%0];" ::"l"(J.p1 + item + 1));
        const int r = it.r;
        const int p0 = (int)(local - it.c0);
        const int p1 = (int)min((long long)it.nin, gend - J.p1_begin - it.c0);
        const bool whole = p0 == 0 && p1 == it.nin;
        double* dst = whole ? J.T + it.t_rel : S + (2 * w + (first ? 0 : 1)) * slot_len;
        const double* in = J.in + it.in_off;
        for (int j0 = 0; j0 < r; j0 += JC) {
            double v[16];
#pragma unroll
            for (int f = 0; f < 16; ++f) v[f] = 0.0;
            const double* wp = J.hb + it.w + (long long)j0 * it.ldw;
            for (int pa = p0 + lane; pa < p1; pa += 64) {
                const int pb = pa + 32;
                const bool okb = pb < p1;
                double wa[JC], wb[JC];
#pragma unroll
                for (int jj = 0; jj < JC; ++jj) {
                    const bool cj = j0 + jj < r;
                    wa[jj] = cj ? __ldg(wp + pa + (long long)jj * it.ldw) : 0.0;
                    wb[jj] = (okb && cj) ? __ldg(wp + pb + (long long)jj * it.ldw) : 0.0;
                }
                const double xa = __ldg(in + pa), xb = okb ? __ldg(in + pb) : 0.0;
#pragma unroll
                for (int jj = 0; jj < JC; ++jj) v[jj] = fma(wb[jj], xb, fma(wa[jj], xa, v[jj]));
            }
            warp_transpose_sum16(v, lane);
            if ((lane & 1) == 0) {
                const int f = lane >> 1;
                if (j0 + f < r) dst[j0 + f] = v[0];
            }
        }
        if (!whole) {
            __threadfence();
            __syncwarp();
            const long long G0 = J.p1_begin + it.c0;
            const long long wa = split_owner(G0, GW, C), wb = split_owner(G0 + it.nin - 1, GW, C);
            int last = 0;
            if (lane == 0) last = atomicAdd(J.cnt1 + item, 1) == (int)(wb - wa);
            last = __shfl_sync(0xffffffffu, last, 0);
            if (last) {
                __threadfence();
                const bool wa_here = split_start(wa, GW, C) == G0;
                double* T = J.T + it.t_rel;
                for (int o = lane; o < r; o += 32) {
                    double t = 0.0;
                    for (long long q = wa; q <= wb; ++q)
                        t += __ldcg(S + piece_slot(q, wa, wa_here) * slot_len + o);
                    T[o] = t;
                }
                if (lane == 0) J.cnt1[item] = 0;
            }
        }
        g = J.p1_begin + it.c0 + p1;
        first = false;
    }
}

// ---------------------------------------------------------------------------
// Phase 2: Y_tile = alpha sum_e A_e B_e + beta Y_tile
// ---------------------------------------------------------------------------
__device__ __forceinline__ double load_a(const double* hb, const P2Entry& e, int i, int p) {
    const double* A = hb + e.a;
    return e.transA ? __ldg(A + p + (long long)i * e.lda) : __ldg(A + i + (long long)p * e.lda);
}

__device__ __forceinline__ void store_out(const JobExec& J, const P2T& it, int i, int c,
                                          double v) {
    double* y = J.out + it.out_off + (it.r0 + i) + (long long)c * J.ldout;
    const double al = J.alpha_scale ? J.alpha * *J.alpha_scale : J.alpha;
    *y = J.beta == 0.0 ? al * v : al * v + J.beta * *y;
}

// One column, tiles of at most 32 rows, a streaming (HBM-bound) kernel.
// Persistent warps stream their share of the tiles' concatenated inner
// dimensions (entry e of a tile covers [cbeg, cbeg + inner)).  Within a
// warp, "column workers" (sub-groups of lanes, one lane per row) split the
// piece evenly and keep U columns of loads in flight.
__global__ void __launch_bounds__(kThreads, 2)
p2_stream_kernel(const JobExec* __restrict__ jobs, int njobs, const JobExec job0, long long C,
                 long long GW, double* __restrict__ S, const int2* __restrict__ start) {
    constexpr int U = 16;
    const int lane = threadIdx.x & 31;
    const long long w = (long long)blockIdx.x * kWarps + (threadIdx.x >> 5);
    if (w >= GW) return;
    constexpr long long slot_len = 32;
    long long g = split_start(w, GW, C);
    const long long gend = split_start(w + 1, GW, C);
    bool first = true;
    // one job with precomputed starts: tiles follow one another
    const bool seq = jobs == nullptr && start != nullptr;
    int tile = 0, ent_first = -1;
    if (seq) {
        const int2 s0 = start[w];
        tile = s0.x;
        ent_first = s0.y;
    }
    while (g < gend) {
        const JobExec& J = jobs ? jobs[find_job(jobs, njobs, g, true)] : job0;
        const long long local = g - J.p2_begin;
        P2T it;
        if (seq) {
            if (!first) {
                do { it = J.p2[++tile]; } while (it.width == 0);
            } else {
                it = J.p2[tile];
            }
        } else {
            tile = 0;
            int hi = J.n2 - 1;
            while (tile < hi) {
                const int mid = (tile + hi + 1) >> 1;
                if (J.p2[mid].c0 <= local) tile = mid;
                else hi = mid - 1;
            }
            it = J.p2[tile];
        }
        const int q0 = (int)(local - it.c0);
        const int q1 = (int)min((long long)it.width, gend - J.p2_begin - it.c0);
        const bool whole = q0 == 0 && q1 == it.width;
        // rows-per-pass RL (power of two <= 32), column sub-groups 32/RL
        int RL = 1;
        while (RL < it.rows && RL < 32) RL <<= 1;
        const int sub = lane / RL, rl = lane % RL, nsub = 32 / RL;
        const bool row_ok = rl < it.rows;
        const int row = it.r0 + rl;
        double acc = 0.0;
        {
            const int chunk = (q1 - q0 + nsub - 1) / nsub;
            int p = q0 + sub * chunk;
            const int pend = min(q1, p + chunk);
            int ei = it.e0;
            if (seq && nsub == 1) {
                if (first) ei = ent_first;
            } else {
                int hi = it.e1 - 1;
                while (ei < hi) {
                    const int mid = (ei + hi + 1) >> 1;
                    if (J.ent[mid].cbeg <= p) ei = mid;
                    else hi = mid - 1;
                }
            }
            while (p < pend) {
                const P2Entry e = J.ent[ei];
                if (ei + 1 < it.e1) asm volatile("prefetch.global.L1 [%0];" ::"l"(J.ent + ei + 1));
                const double* EB = e.b_from_t ? J.T + e.b_off : J.in + e.b_off;
                const int stop = min(pend, e.cbeg + e.inner);
                int q = p - e.cbeg;                 // column within the entry
                const int qstop = stop - e.cbeg;
                for (; q + U - 1 < qstop; q += U) {
                    double av[U], bv[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        bv[u] = __ldg(EB + (q + u));
                        av[u] = row_ok ? load_a(J.hb, e, row, q + u) : 0.0;
                    }
#pragma unroll
                    for (int u = 0; u < U; ++u) acc = fma(av[u], bv[u], acc);
                }
                for (; q < qstop; ++q) {
                    const double av = row_ok ? load_a(J.hb, e, row, q) : 0.0;
                    acc = fma(av, __ldg(EB + q), acc);
                }
                p = stop;
                ++ei;
            }
        }
        // reduce over the column sub-groups (lanes with equal rl)
        for (int o = 16; o >= RL; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (whole) {
            if (sub == 0 && row_ok) store_out(J, it, rl, 0, acc);
        } else {
            double* P = S + (2 * w + (first ? 0 : 1)) * slot_len;
            if (sub == 0 && row_ok) P[rl] = acc;
            __threadfence();
            __syncwarp();
            const long long G0 = J.p2_begin + it.c0;
            const long long wa = split_owner(G0, GW, C), wb = split_owner(G0 + it.width - 1, GW, C);
            int last = 0;
            if (lane == 0) last = atomicAdd(J.cnt2 + tile, 1) == (int)(wb - wa);
            last = __shfl_sync(0xffffffffu, last, 0);
            if (last) {
                __threadfence();
                const bool wa_here = split_start(wa, GW, C) == G0;
                for (int i = lane; i < it.rows; i += 32) {
                    double t = 0.0;
                    for (long long q = wa; q <= wb; ++q)
                        t += __ldcg(S + piece_slot(q, wa, wa_here) * slot_len + i);
                    store_out(J, it, i, 0, t);
                }
                if (lane == 0) J.cnt2[tile] = 0;
            }
        }
        g = J.p2_begin + it.c0 + q1;
        first = false;
    }
}

// Row tiles without entries, over all jobs of a launch (list of (job, tile)):
// output = beta * output (alpha times an empty sum).
__global__ void p2_zero_kernel(const JobExec* __restrict__ jobs, const JobExec job0,
                               const int2* __restrict__ list, int n) {
    for (int t = blockIdx.x; t < n; t += gridDim.x) {
        const int2 jt = list[t];
        const JobExec& J = jobs ? jobs[jt.x] : job0;
        const P2T it = J.p2[jt.y];
        for (int o = threadIdx.x; o < it.rows * J.k; o += blockDim.x)
            store_out(J, it, o % it.rows, o / it.rows, 0.0);
    }
}

// One launch for the tiles without entries of every job.
void launch_zero_tiles(Context& ctx, const std::vector<std::shared_ptr<JobTemplate>>& tmpl,
                       const std::vector<MatJob>& jobs, const JobExec* jobs_d, const JobExec& job0) {
    std::vector<int2> list;
    int j = 0;
    for (size_t i = 0; i < jobs.size(); ++i) {
        if (jobs[i].k == 0) continue;
        for (int t : tmpl[i]->hzero) list.push_back(make_int2(j, t));
        ++j;
    }
    if (list.empty()) return;
    DeviceBuffer<int2> d;
    d.upload(list, ctx.stream);
    LaunchScope ls(ctx, "hmm_zero_tiles");
    p2_zero_kernel<<<std::min((int)list.size(), 4 * ctx.num_sms), 256, 0, ctx.stream>>>(
        jobs_d, job0, d.get(), (int)list.size());
    HMB_CHECK_LAUNCH();
}

// ---------------------------------------------------------------------------
// TF32, many columns: 64 x 64 output tiles, 4 warps of 32 x 32 each; operands
// staged through shared memory in chunks of KC inner indices by cp.async, two
// stages (the next chunk loads while this one is multiplied).
// ---------------------------------------------------------------------------
constexpr int WT = kWideTile;   // tile rows = tile columns
constexpr int KC = 16;          // inner chunk
constexpr int WTHREADS = 128;   // 2 x 2 warps of 32 x 32
constexpr int SP = WT + 8;      // smem row: fragment loads hit 32 distinct banks

constexpr int NSTAGE = 2;       // chunk buffers per CTA
struct WideSmem32 {
    float a[NSTAGE][KC][SP];   // a[buf][p][i] = A(i, p)
    float b[NSTAGE][KC][SP];   // b[buf][p][c] = B(p, c)
};

// The copies carry no "memory" clobber: their shared-memory destinations are
// read only after cp_async_wait (which has one) and a barrier, and without
// it the compiler may keep the work-list fields that address the copies in
// registers instead of reloading them from global memory after every copy.
__device__ __forceinline__ void cp_async4(float* dst, const float* src, bool valid) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src),
                 "r"(valid ? 4 : 0));
}

// TF32 tensor-core MMA 16 x 8 x 8, FP32 accumulation.  Fragments (g = lane/4,
// t = lane%4): A a0 (g, t), a1 (g+8, t), a2 (g, t+4), a3 (g+8, t+4); B b0 (t, g),
// b1 (t+4, g); C c0 (g, 2t), c1 (g, 2t+1), c2 (g+8, 2t), c3 (g+8, 2t+1).
__device__ __forceinline__ void tmma(float* d, const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
        "{%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__device__ __forceinline__ float round_tf32(double x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"((float)x));
    return __uint_as_float(r);
}

// TF32 tiles: slot s = ((mb * 4 + nb) * 4 + e) of MMA block (mb, nb) (16 x 8)
// of the warp's 32 x 32 quarter, C fragment element e.
__device__ __forceinline__ int acc_row_tf(int s, int warp, int lane) {
    return (warp & 1) * 32 + (s >> 4) * 16 + (lane >> 2) + ((s & 2) ? 8 : 0);
}
__device__ __forceinline__ int acc_col_tf(int s, int warp, int lane) {
    return (warp >> 1) * 32 + ((s >> 2) & 3) * 8 + 2 * (lane & 3) + (s & 1);
}

__device__ __forceinline__ void wide_mma_tf(const WideSmem32& sm, int buf, int warp, int lane,
                                            float (&acc)[32]) {
    const int g = lane >> 2, t = lane & 3;
    const int r0 = (warp & 1) * 32 + g, c0 = (warp >> 1) * 32 + g;
#pragma unroll
    for (int kb = 0; kb < KC; kb += 8) {
        uint32_t a[2][4], b[4][2];
#pragma unroll
        for (int mb = 0; mb < 2; ++mb) {
            a[mb][0] = __float_as_uint(sm.a[buf][kb + t][r0 + mb * 16]);
            a[mb][1] = __float_as_uint(sm.a[buf][kb + t][r0 + mb * 16 + 8]);
            a[mb][2] = __float_as_uint(sm.a[buf][kb + t + 4][r0 + mb * 16]);
            a[mb][3] = __float_as_uint(sm.a[buf][kb + t + 4][r0 + mb * 16 + 8]);
        }
#pragma unroll
        for (int nb = 0; nb < 4; ++nb) {
            b[nb][0] = __float_as_uint(sm.b[buf][kb + t][c0 + nb * 8]);
            b[nb][1] = __float_as_uint(sm.b[buf][kb + t + 4][c0 + nb * 8]);
        }
#pragma unroll
        for (int mb = 0; mb < 2; ++mb)
#pragma unroll
            for (int nb = 0; nb < 4; ++nb) tmma(&acc[(mb * 4 + nb) * 4], a[mb], b[nb]);
    }
}

// B chunk: B(p, c) = Bp[p + c * ldb] for p < len, c < cols (p fastest).
__device__ __forceinline__ void load_b_chunk(WideSmem32& sm, int buf, const float* Bp, int ldb,
                                             int len, int cols, int tid) {
#pragma unroll
    for (int e = tid; e < KC * WT; e += WTHREADS) {
        const int p = e % KC, c = e / KC;
        const bool v = p < len && c < cols;
        cp_async4(&sm.b[buf][p][c], v ? Bp + p + (long long)c * ldb : Bp, v);
    }
}

// The wide kernels stream a sequence of KC-chunks: phase 1 the chunks of
// every W1 tile (its nin input rows), phase 2 the chunks of every row tile's
// entries (no chunk spans two entries), over all jobs.  A persistent CTA takes
// an even share [b C / G, (b+1) C / G) of the sequence; the next chunk (of the
// same or the next tile) loads while the current one is multiplied.  A tile
// whose chunks a CTA holds completely is written directly; a tile cut between
// CTAs b_a..b_b leaves 64 x 64 partials (slot 2b for a CTA's first piece,
// 2b + 1 for its last) that the piece finishing last adds up in CTA order.
struct ChunkPos {
    int job, tile, ei, pos;   // phase 1: ei unused, pos = row offset in the tile's input
};

template <int PHASE>
__device__ __forceinline__ int tiles_of(const JobExec& J) { return PHASE == 1 ? J.n1 : J.n2; }
template <int PHASE>
__device__ __forceinline__ const int* chunk_prefix(const JobExec& J) { return PHASE == 1 ? J.w1cp : J.tcp; }

// The TF32 form: FP32 copy of the blocks and of the input, TF32 tensor-core
// MMA, FP32 accumulation, FP64 output.
template <int PHASE>
__global__ void __launch_bounds__(WTHREADS, 4)
wide_tf32_kernel(const JobExec* __restrict__ jobs, int njobs, const JobExec job0, long long C, int G) {
    extern __shared__ __align__(16) unsigned char wide_smem[];
    WideSmem32& sm = *reinterpret_cast<WideSmem32*>(wide_smem);
    __shared__ int last_flag;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int b = blockIdx.x, y = blockIdx.y;
    const long long g0 = split_start(b, G, C), g1 = split_start(b + 1, G, C);
    if (g0 >= g1) return;
    auto job = [&](int j) -> const JobExec& { return jobs ? jobs[j] : job0; };
    // locate the first chunk
    ChunkPos cur{};
    {
        cur.job = jobs ? find_job(jobs, njobs, g0, PHASE == 2) : 0;
        const JobExec& J = job(cur.job);
        const long long local = g0 - (PHASE == 1 ? J.p1_begin : J.p2_begin);
        const int* cp = chunk_prefix<PHASE>(J);
        int lo = 0, hi = tiles_of<PHASE>(J) - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (cp[mid] <= local) lo = mid;
            else hi = mid - 1;
        }
        // skip tiles without chunks
        while (cp[lo + 1] <= local) ++lo;
        cur.tile = lo;
        const int kin = (int)(local - cp[lo]);
        if (PHASE == 1) {
            cur.pos = kin * KC;
        } else {
            const P2T it = J.p2[lo];
            int e = it.e0, eh = it.e1 - 1;
            while (e < eh) {
                const int mid = (e + eh + 1) >> 1;
                if (J.ekc[mid] <= kin) e = mid;
                else eh = mid - 1;
            }
            cur.ei = e;
            cur.pos = (kin - J.ekc[e]) * KC;
        }
    }
    // loads the chunk at `c` into buffer `buf`; returns whether it is the last
    // chunk of its tile; advances `c`
    auto load = [&](ChunkPos& c, int buf) -> bool {
        const JobExec& J = job(c.job);
        const int cols = min(WT, J.k - y * WT);
        bool last;
        if (PHASE == 1) {
            const W1Tile* t = J.w1 + c.tile;
            const int len = min(KC, t->nin - c.pos), rows = t->rows;
#pragma unroll
            for (int e = tid; e < WT * KC; e += WTHREADS) {
                const int p = e % KC, i = e / KC;   // W columns are contiguous
                const bool v = p < len && i < rows;
                const long long wo = t->wcol[v ? i : 0];
                const float* w0 = J.hb32 + wo;
                cp_async4(&sm.a[buf][p][i], v ? w0 + c.pos + p : w0, v);
            }
            load_b_chunk(sm, buf, J.in32 + t->in_off + c.pos + (long long)y * WT * J.ldin32,
                         J.ldin32, len, cols, tid);
            c.pos += len;
            last = c.pos >= t->nin;
        } else {
            const P2T it = J.p2[c.tile];
            const P2Entry e = J.ent[c.ei];
            const int len = min(KC, e.inner - c.pos);
            const float* Eb = J.hb32 + e.a;
            if (!e.transA) {
                const float* A = Eb + it.r0 + (long long)c.pos * e.lda;
#pragma unroll
                for (int x = tid; x < WT * KC; x += WTHREADS) {
                    const int i = x % WT, p = x / WT;   // rows contiguous
                    const bool v = p < len && i < it.rows;
                    cp_async4(&sm.a[buf][p][i], v ? A + i + (long long)p * e.lda : Eb, v);
                }
            } else {
                const float* A = Eb + c.pos + (long long)it.r0 * e.lda;
#pragma unroll
                for (int x = tid; x < WT * KC; x += WTHREADS) {
                    const int p = x % KC, i = x / KC;   // inner index contiguous
                    const bool v = p < len && i < it.rows;
                    cp_async4(&sm.a[buf][p][i], v ? A + p + (long long)i * e.lda : Eb, v);
                }
            }
            const float* EB;
            int ldb;
            if (e.b_from_t) { EB = J.T32 + e.b_off * J.k; ldb = e.ldt; }
            else { EB = J.in32 + e.b_off; ldb = J.ldin32; }
            load_b_chunk(sm, buf, EB + c.pos + (long long)y * WT * ldb, ldb, len, cols, tid);
            c.pos += len;
            last = false;
            if (c.pos >= e.inner) {
                c.pos = 0;
                ++c.ei;
                last = c.ei >= it.e1;
            }
        }
        cp_async_commit();
        if (last) {   // move to the next tile with chunks (possibly of the next job)
            c.pos = 0;
            for (;;) {
                ++c.tile;
                if (c.tile >= tiles_of<PHASE>(job(c.job))) {
                    if (!jobs || c.job + 1 >= njobs) break;
                    ++c.job;
                    c.tile = -1;
                    continue;
                }
                const int* cp = chunk_prefix<PHASE>(job(c.job));
                if (cp[c.tile + 1] > cp[c.tile]) break;
            }
            if (PHASE == 2 && c.tile < tiles_of<PHASE>(job(c.job))) c.ei = job(c.job).p2[c.tile].e0;
        }
        return last;
    };
    float acc[32];
#pragma unroll
    for (int q = 0; q < 32; ++q) acc[q] = 0;
    auto arow = [&](int k) { return acc_row_tf(k, warp, lane); };
    auto acol = [&](int k) { return acc_col_tf(k, warp, lane); };
    // NSTAGE-deep ring: chunk q sits in buffer q % NSTAGE and is issued
    // NSTAGE - 1 chunks ahead; one commit group per chunk slot (empty past
    // the end) keeps the wait count constant
    ChunkPos loaded[NSTAGE];
    bool lastc[NSTAGE];
    const long long n = g1 - g0;
#pragma unroll
    for (int s = 0; s < NSTAGE - 1; ++s) {
        if (s < n) {
            loaded[s] = cur;
            lastc[s] = load(cur, s);
        } else {
            cp_async_commit();
        }
    }
    bool first_piece = true;
    for (long long q = 0; q < n; ++q) {
        const long long qn = q + NSTAGE - 1;
        const int bn = (int)(qn % NSTAGE);
        if (qn < n) {
            loaded[bn] = cur;
            lastc[bn] = load(cur, bn);
        } else {
            cp_async_commit();
        }
        cp_async_wait<NSTAGE - 1>();
        __syncthreads();
        const int buf = (int)(q % NSTAGE);
        wide_mma_tf(sm, buf, warp, lane, acc);
        __syncthreads();
        if (!lastc[buf] && q + 1 < n) continue;
        // flush the tile of this chunk
        const ChunkPos& t = loaded[buf];
        const JobExec& J = job(t.job);
        const int cols = min(WT, J.k - y * WT);
        const long long base = PHASE == 1 ? J.p1_begin : J.p2_begin;
        const int* cp = chunk_prefix<PHASE>(J);
        const long long T0 = base + cp[t.tile], T1 = base + cp[t.tile + 1];
        const bool whole = T0 >= g0 && T1 <= g1;
        int rows;
        const W1Tile* wt = nullptr;
        P2T it{};
        if (PHASE == 1) {
            wt = J.w1 + t.tile;
            rows = wt->rows;
        } else {
            it = J.p2[t.tile];
            rows = it.rows;
        }
        auto emit = [&](int i, int c, double v) {
            if (PHASE == 1) {
                const long long o = wt->trel[i] * J.k + wt->tj[i] + (long long)(y * WT + c) * wt->tr[i];
                J.T32[o] = round_tf32(v);
            } else {
                store_out(J, it, i, y * WT + c, v);
            }
        };
        if (whole && PHASE == 1) {
            // the thread's 32 accumulators lie in 4 tile rows: their T
            // offsets are loaded once, before the stores (which the compiler
            // must otherwise assume may change them)
            auto rslot = [](int k) { return ((k >> 4) << 1) | ((k >> 1) & 1); };
            long long rbase[4], rstep[4];
            const long long kk = J.k;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int i = arow(((q >> 1) << 4) | ((q & 1) << 1));
                const bool ok = i < rows;
                rbase[q] = ok ? wt->trel[i] * kk + wt->tj[i] : 0;
                rstep[q] = ok ? (long long)wt->tr[i] : 0;
            }
            float* T32p = J.T32;
#pragma unroll
            for (int k = 0; k < 32; ++k) {
                const int i = arow(k), c = acol(k);
                if (i < rows && c < cols) {
                    const long long o = rbase[rslot(k)] + (long long)(y * WT + c) * rstep[rslot(k)];
                    T32p[o] = round_tf32((double)acc[k]);
                }
            }
        } else if (whole) {
#pragma unroll
            for (int k = 0; k < 32; ++k) {
                const int i = arow(k), c = acol(k);
                if (i < rows && c < cols) emit(i, c, (double)acc[k]);
            }
        } else {
            double* part = J.part + ((long long)y * 2 * G) * (WT * WT);
            double* mine = part + (2LL * b + (first_piece ? 0 : 1)) * (WT * WT);
#pragma unroll
            for (int k = 0; k < 32; ++k) mine[arow(k) + WT * acol(k)] = (double)acc[k];
            __threadfence();
            __syncthreads();
            const long long wa = split_owner(T0, G, C), wb = split_owner(T1 - 1, G, C);
            int* cnt = (PHASE == 1 ? J.cnt1 : J.cnt2) + (long long)t.tile * gridDim.y + y;
            if (tid == 0) last_flag = atomicAdd(cnt, 1) == (int)(wb - wa);
            __syncthreads();
            if (last_flag) {
                __threadfence();
                const bool wa_here = split_start(wa, G, C) == T0;
                for (int x = tid; x < rows * cols; x += WTHREADS) {
                    const int i = x % rows, c = x / rows;
                    double v = 0.0;
                    for (long long w = wa; w <= wb; ++w)
                        v += __ldcg(part + piece_slot(w, wa, wa_here) * (WT * WT) + i + WT * c);
                    emit(i, c, v);
                }
                if (tid == 0) *cnt = 0;
            }
            __syncthreads();
        }
#pragma unroll
        for (int k = 0; k < 32; ++k) acc[k] = 0;
        first_piece = false;
    }
}

// ---------------------------------------------------------------------------
// FP64, two columns and more: 64-row x NT-column tiles, NT = 8, 16, 32 or 64,
// on the FP64 tensor cores (mma.m8n8k4.f64), 128 threads.
//
// Bound by the FP64 tensor pipe from about 40 columns on, by HBM below.  The
// operands of a chunk (16 inner indices) reach shared memory by 16-byte
// cp.async two chunks ahead, in the order memory has them: an operand whose
// inner index is contiguous (W, the input, T, the transposed dense leaves) as
// rows of 16 inner indices, their eight 16-byte units exchanged between halves
// on odd rows; the others (U, the dense leaves) as columns of 64 rows with a
// stride of 66.  Either way the copies and the fragment loads touch each bank
// once, and a fragment load serves two MMAs: the inner index of the first is
// 2t, of the second 2t + 1 (t = lane % 4), for both operands.  (Copies of 8
// bytes into one common layout, whose bank conflicts took 30 % of the time,
// and the work-list reads in front of every chunk held the earlier kernel to
// 23 % and 38 % of the pipe.)  The chunks are described by a flat list, read
// two chunks ahead: a rank-16 factor is one chunk, so every chunk brings new
// addresses.  A warp whose rows or columns all lie beyond the tile does not
// multiply; testing that per 8 x 8 block cost more than the blocks (128
// columns of the 200 x 184 operator: 5 %).  Measured, 64 columns of the 128 x
// 128 operator (rank 16): 392 -> 227 us for both phases, 19 TF/s of 37; 5
// columns of the 117 x 101 one, transposed: 147 -> 74 us.
// ---------------------------------------------------------------------------
template <int NT>
struct Tile64 {
    static constexpr int WN = NT == 64 ? 2 : 1, WM = 4 / WN;   // warps along columns, rows
    static constexpr int MB = 8 / WM, NB = NT / (8 * WN);      // 8 x 8 blocks of a warp
    static constexpr int STAGES = 3;
    // CTAs an SM: fewer for the wide tiles, whose accumulators and addresses
    // otherwise spill (when 64 columns of the 128 x 128 operator took 283 us:
    // 4 CTAs 300 us, 4 stages 290 us; when 5 columns of the 117 x 101 one took
    // 82 us: 5 CTAs 88 us)
    static constexpr int CTAS = NT == 64 ? 3 : NT == 32 ? 4 : 6;
    static constexpr int ASZ = KC * 66;                        // doubles of an A stage
    static constexpr int BSZ = NT * KC;
    static constexpr size_t smem = (size_t)STAGES * (ASZ + BSZ) * sizeof(double);
};

__device__ __forceinline__ bool even16(const double* p, long long stride) {
    return ((reinterpret_cast<size_t>(p) | (size_t)(stride << 3)) & 15) == 0;
}

// ONE: a single job, whose description is a kernel parameter (constant memory)
// and not a list in global memory.
template <int PHASE, int NT, bool ONE>
__global__ void __launch_bounds__(WTHREADS, Tile64<NT>::CTAS)
wide64_kernel(const JobExec* __restrict__ jobs, int njobs, const JobExec job0, long long C, int G) {
    using TL = Tile64<NT>;
    constexpr int MB = TL::MB, NB = TL::NB, WM = TL::WM, WN = TL::WN, ST = TL::STAGES;
    extern __shared__ __align__(16) unsigned char wide_smem[];
    double* const As = reinterpret_cast<double*>(wide_smem);
    double* const Bs = As + ST * TL::ASZ;
    // per stage: job, tile, inner indices | layout << 8 | last chunk << 9, rows | columns << 8
    __shared__ int4 meta[ST];
    __shared__ int last_flag;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int wm = warp % WM, wn = warp / WM;
    const int b = blockIdx.x, y = blockIdx.y;
    const long long g0 = split_start(b, G, C), g1 = split_start(b + 1, G, C);
    if (g0 >= g1) return;
    auto job = [&](int j) -> const JobExec& {
        if constexpr (ONE) return job0;
        else return jobs[j];
    };

    // ---- the chunk to be loaded next: this thread's addresses --------------
    const int ku = tid & 7, kr = tid >> 3;     // unit and row of an inner-contiguous copy
    const int mu = tid & 31, mp = tid >> 5;    // unit and column of a row-contiguous copy
    const unsigned as0 = (unsigned)__cvta_generic_to_shared(As);
    const unsigned bs0 = (unsigned)__cvta_generic_to_shared(Bs);
    const unsigned dk = (unsigned)(kr * KC + 2 * (ku ^ ((kr & 1) << 2))) * 8;
    const unsigned dm = (unsigned)(mp * 66 + 2 * mu) * 8;
    int cj = ONE ? 0 : find_job(jobs, njobs, g0, PHASE == 2);
    long long gn = g0, jend = 0;   // index of the chunk in `next`; end of its job
    auto begin_of = [&](int j) { return PHASE == 1 ? job(j).p1_begin : job(j).p2_begin; };
    if (!ONE) jend = cj + 1 < njobs ? begin_of(cj + 1) : C;
    int nj = cj;                   // job of `next`
    WideChunk next;                // the chunk after the one whose addresses are ready
    auto fetch_next = [&]() {
        if (gn >= g1) return;
        if (!ONE)
            while (gn >= jend) {
                ++nj;
                jend = nj + 1 < njobs ? begin_of(nj + 1) : C;
            }
        const JobExec& J = job(nj);
        const int4* p = reinterpret_cast<const int4*>((PHASE == 1 ? J.ch1 : J.ch2) + (gn - begin_of(nj)));
        const int4 u = __ldg(p), v = __ldg(p + 1);
        next.a = (long long)(((unsigned long long)(unsigned)u.y << 32) | (unsigned)u.x);
        next.lda = u.z;
        next.b = u.w;
        next.pos = v.x;
        next.ldt = v.y;
        next.tile = v.z;
        next.bits = v.w;
        ++gn;
    };
    int ctile = -1, cbits = 0, cols = 0, lda = 0, ldb = 0;
    bool a16 = false, b16 = false;
    const double *pa = nullptr, *pb = nullptr, *any = nullptr;
    long long wo[4];                           // phase 1: this thread's columns of W
    unsigned wo16 = 0;
    // the addresses of `next`, which becomes the current chunk
    auto advance = [&]() {
        const bool new_tile = next.tile != ctile || (!ONE && nj != cj);
        cj = nj;
        const JobExec& J = job(cj);
        any = J.hb;
        ctile = next.tile;
        cbits = next.bits;
        cols = min(NT, J.k - y * NT);
        if (PHASE == 1) {
            if (new_tile) {
                const W1Tile* w = J.w1 + ctile;
                const int rows = cbits >> 16;
                wo16 = 0;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    wo[q] = __ldg(w->wcol + min(kr + 16 * q, rows - 1));
                    wo16 |= (wo[q] & 1) ? 0u : 1u << q;
                    wo[q] += 2 * ku;
                }
            }
            pa = J.hb + next.pos;
            ldb = J.ldin;
            pb = J.in + next.b + next.pos;
        } else {
            lda = next.lda;
            const bool km = (cbits & 256) != 0;
            pa = J.hb + next.a;
            a16 = ((next.a | lda) & 1) == 0;   // the storage itself is aligned
            pa += (long long)(km ? kr : mp) * lda + 2 * (km ? ku : mu);
            ldb = next.ldt > 0 ? next.ldt : J.ldin;
            pb = (next.ldt > 0 ? J.T + (long long)next.b * J.k : J.in + next.b) + next.pos;
        }
        b16 = even16(pb, ldb);
        pb += (long long)(y * NT + kr) * ldb + 2 * ku;
        fetch_next();
    };
    fetch_next();
    advance();
    // copies the current chunk to stage `buf` and moves on
    auto load = [&](int buf) {
        const int len = cbits & 255, rows = cbits >> 16;
        const unsigned A = as0 + (unsigned)buf * (TL::ASZ * 8), B = bs0 + (unsigned)buf * (TL::BSZ * 8);
        const int kbytes = max(0, min(16, (len - 2 * ku) * 8));
        if (PHASE == 1) {
#pragma unroll
            for (int q = 0; q < 4; ++q)
                copy_pair(A + dk + q * (16 * KC * 8), pa + wo[q], kr + 16 * q < rows ? kbytes : 0,
                          (wo16 >> q) & 1, any);
        } else {
            const bool km = (cbits & 256) != 0;
            const int bytes = km ? kbytes : max(0, min(16, (rows - 2 * mu) * 8));
            const int lim = km ? (rows - kr + 15) >> 4 : (len - mp + 3) >> 2;
            const unsigned d = A + (km ? dk : dm), ds = km ? 16 * KC * 8 : 4 * 66 * 8;
            const long long sa = (long long)lda << (km ? 4 : 2);
            const double* src = pa;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                copy_pair(d + q * ds, src, q < lim ? bytes : 0, a16, any);
                src += sa;
            }
        }
        if (NT >= 16 || kr < NT) {
            const double* src = pb;
            const long long sb = (long long)ldb << 4;
#pragma unroll
            for (int q = 0; q < (NT + 15) / 16; ++q) {
                copy_pair(B + dk + q * (16 * KC * 8), src, kr + 16 * q < cols ? kbytes : 0, b16, any);
                src += sb;
            }
        }
        cp_async_commit();
        if (tid == 0) meta[buf] = make_int4(cj, ctile, cbits & 0xffff, rows | cols << 8);
        advance();   // (past the last chunk: the same addresses again, unused)
    };

    double acc[MB][NB][2];
#pragma unroll
    for (int m = 0; m < MB; ++m)
#pragma unroll
        for (int n = 0; n < NB; ++n) acc[m][n][0] = acc[m][n][1] = 0.0;
    const long long n = g1 - g0;
#pragma unroll
    for (int s = 0; s < ST - 1; ++s) {
        if (s < n) load(s);
        else cp_async_commit();
    }
    const int unit = ((g & 1) << 2) ^ t;   // this lane's swizzled unit of an even half row
    bool first_piece = true;
    int buf = 0;
    for (long long q = 0; q < n; ++q) {
        cp_async_wait<ST - 2>();
        __syncthreads();
        // every warp is done with the stage before: refill it
        if (q + ST - 1 < n) load(buf == 0 ? ST - 1 : buf - 1);
        else cp_async_commit();
        const int4 mt = meta[buf];
        const int len = mt.z & 255;
        const int trows = mt.w & 255, tcols = mt.w >> 8;
        // a warp whose blocks all lie beyond the tile has nothing to multiply
        const bool live = 8 * wm < trows && 8 * wn < tcols;
        const double* A = As + buf * TL::ASZ;
        const double* B = Bs + buf * TL::BSZ;
        buf = buf + 1 == ST ? 0 : buf + 1;
#pragma unroll
        for (int kp = 0; kp < KC / 8; ++kp) {
            if (!live || 8 * kp >= len) break;
            double2 a[MB], x[NB];
            if (PHASE == 1 || (mt.z & 256)) {
#pragma unroll
                for (int m = 0; m < MB; ++m)
                    a[m] = *reinterpret_cast<const double2*>(
                        A + (8 * (WM * m + wm) + g) * KC + 2 * (unit ^ (4 * kp)));
            } else {
#pragma unroll
                for (int m = 0; m < MB; ++m) {
                    const double* p = A + (8 * kp + 2 * t) * 66 + 8 * (WM * m + wm) + g;
                    a[m].x = p[0];
                    a[m].y = p[66];
                }
            }
#pragma unroll
            for (int c = 0; c < NB; ++c)
                x[c] = *reinterpret_cast<const double2*>(
                    B + (8 * (WN * c + wn) + g) * KC + 2 * (unit ^ (4 * kp)));
#pragma unroll
            for (int m = 0; m < MB; ++m)
#pragma unroll
                for (int c = 0; c < NB; ++c) dmma(acc[m][c], a[m].x, x[c].x);
#pragma unroll
            for (int m = 0; m < MB; ++m)
#pragma unroll
                for (int c = 0; c < NB; ++c) dmma(acc[m][c], a[m].y, x[c].y);
        }
        if (!(mt.z & 512) && q + 1 < n) continue;
        // ---- the tile (or this CTA's piece of it) is complete -------------
        const JobExec& J = job(mt.x);
        const long long base = PHASE == 1 ? J.p1_begin : J.p2_begin;
        const int* cp = chunk_prefix<PHASE>(J);
        const long long T0 = base + cp[mt.y], T1 = base + cp[mt.y + 1];
        const bool whole = T0 >= g0 && T1 <= g1;
        const W1Tile* wt = PHASE == 1 ? J.w1 + mt.y : nullptr;
        P2T it{};
        if (PHASE == 2) it = J.p2[mt.y];
        // one row of the tile's blocks (m of this warp) to where it belongs
        auto store_row = [&](int m, const double (&v)[NB][2]) {
            const int i = 8 * (WM * m + wm) + g;
            if (i >= trows) return;
            long long rbase = 0, rstep = 0;
            if (PHASE == 1) {
                rbase = wt->trel[i] * J.k + wt->tj[i];
                rstep = wt->tr[i];
            }
#pragma unroll
            for (int c = 0; c < NB; ++c)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int col = 8 * (WN * c + wn) + 2 * t + h;
                    if (col >= tcols) continue;
                    if (PHASE == 1) J.T[rbase + (long long)(y * NT + col) * rstep] = v[c][h];
                    else store_out(J, it, i, y * NT + col, v[c][h]);
                }
        };
        if (whole) {
#pragma unroll
            for (int m = 0; m < MB; ++m) store_row(m, acc[m]);
        } else {
            // Partials in the order of the accumulators, 16 bytes a thread; blocks
            // beyond the tile are neither written nor read.  The last piece adds
            // all of them in CTA order.  Bound by the latency of its loads, so
            // several CTAs' partials are in flight for a block row, for the
            // 8-column tiles for both block rows of a warp, within the registers
            // of the main loop (whose spills cost more than this saves: all loads
            // of four CTAs first, 8 columns of the 128 x 128 operator 114 us
            // against 90).  One element after the other, 64 columns: 16 x 16
            // points of rank 4 (16 pieces a tile) 141 -> 19 us, 128 x 128 points
            // of rank 16 284 -> 227 us.
            auto in_tile = [&](int m, int c) {
                return 8 * (WM * m + wm) < trows && 8 * (WN * c + wn) < tcols;
            };
            double2* part = reinterpret_cast<double2*>(J.part) + ((long long)y * 2 * G) * (WT * NT / 2) + tid;
            double2* mine = part + (2LL * b + (first_piece ? 0 : 1)) * (WT * NT / 2);
#pragma unroll
            for (int m = 0; m < MB; ++m)
#pragma unroll
                for (int c = 0; c < NB; ++c)
                    if (in_tile(m, c))
                        mine[(m * NB + c) * WTHREADS] = make_double2(acc[m][c][0], acc[m][c][1]);
            __threadfence();
            __syncthreads();
            const long long wa = split_owner(T0, G, C), wb = split_owner(T1 - 1, G, C);
            int* cnt = (PHASE == 1 ? J.cnt1 : J.cnt2) + (long long)mt.y * gridDim.y + y;
            if (tid == 0) last_flag = atomicAdd(cnt, 1) == (int)(wb - wa);
            __syncthreads();
            if (last_flag) {
                __threadfence();
                const bool wa_here = split_start(wa, G, C) == T0;
                constexpr int MG = NT == 8 ? MB : 1;   // block rows at a time
#pragma unroll 1
                for (int m0 = 0; m0 < MB && 8 * (WM * m0 + wm) < trows; m0 += MG) {
                    double v[MG][NB][2];
#pragma unroll
                    for (int m = 0; m < MG; ++m)
#pragma unroll
                        for (int c = 0; c < NB; ++c) v[m][c][0] = v[m][c][1] = 0.0;
#pragma unroll(NT == 16 ? (ONE ? 2 : 1) : 4)
                    for (long long w = wa; w <= wb; ++w) {
                        const double2* p =
                            part + piece_slot(w, wa, wa_here) * (WT * NT / 2) + m0 * NB * WTHREADS;
#pragma unroll
                        for (int m = 0; m < MG; ++m)
#pragma unroll
                            for (int c = 0; c < NB; ++c)
                                if (in_tile(m0 + m, c)) {
                                    const double2 x = __ldcg(p + (m * NB + c) * WTHREADS);
                                    v[m][c][0] += x.x;
                                    v[m][c][1] += x.y;
                                }
                    }
#pragma unroll
                    for (int m = 0; m < MG; ++m) store_row(m0 + m, v[m]);
                }
                if (tid == 0) *cnt = 0;
            }
        }
#pragma unroll
        for (int m = 0; m < MB; ++m)
#pragma unroll
            for (int c = 0; c < NB; ++c) acc[m][c][0] = acc[m][c][1] = 0.0;
        first_piece = false;
    }
}

// The W1 tiles (CTAs 0 .. nw1 - 1) with their chunks, and the chunks of the row
// tiles (the CTAs after them).
__global__ void expand_template_kernel(const W1Source* __restrict__ src, int nw1, const P1T* __restrict__ p1,
                                       const P2T* __restrict__ p2, int n2, const P2Entry* __restrict__ ent,
                                       const int* __restrict__ prefix, W1Tile* __restrict__ w1,
                                       WideChunk* __restrict__ chunks) {
    const int* w1cp = prefix;
    const int* tcp = prefix + nw1 + 1;
    const int* ekc = tcp + n2 + 1;
    const int tid = threadIdx.x, t = blockIdx.x;
    if (t < nw1) {
        const W1Source s = src[t];
        W1Tile& w = w1[t];
        if (tid == 0) {
            w.in_off = s.in_off;
            w.nin = s.nin;
            w.rows = s.rows;
        }
        for (int i = tid; i < kWideTile; i += blockDim.x) {
            long long wcol = 0, trel = 0;
            int tj = 0, tr = 0;
            if (i < s.rows) {
                int it = s.item;
                tj = s.col + i;
                while (tj >= (tr = p1[it].r)) {
                    tj -= tr;
                    ++it;
                }
                wcol = p1[it].w + (long long)tj * p1[it].ldw;
                trel = p1[it].t_rel;
            }
            w.wcol[i] = wcol;
            w.trel[i] = trel;
            w.tj[i] = tj;
            w.tr[i] = tr;
        }
        WideChunk* c = chunks + w1cp[t];
        for (int pos = tid * KC; pos < s.nin; pos += (int)blockDim.x * KC)
            c[pos / KC] = {0, 0, (int)s.in_off, pos, 0, t,
                           min(KC, s.nin - pos) | 256 | (pos + KC >= s.nin ? 512 : 0) | s.rows << 16};
        return;
    }
    const int u = t - nw1;
    const P2T it = p2[u];
    for (int e = it.e0 + tid; e < it.e1; e += blockDim.x) {
        const P2Entry E = ent[e];
        WideChunk* c = chunks + w1cp[nw1] + tcp[u] + ekc[e];
        for (int pos = 0; pos < E.inner; pos += KC) {
            const long long a = E.a + (E.transA ? pos + (long long)it.r0 * E.lda
                                                : it.r0 + (long long)pos * E.lda);
            c[pos / KC] = {a, E.lda, (int)E.b_off, pos, E.b_from_t ? E.ldt : 0, u,
                           min(KC, E.inner - pos) | (E.transA ? 256 : 0) |
                               (e + 1 == it.e1 && pos + KC >= E.inner ? 512 : 0) | it.rows << 16};
        }
    }
}

// Work lists of one subtree of one H-matrix.
std::shared_ptr<JobTemplate> build_template(Context& ctx, const HMatrix& H, int root,
                                            bool trans, int row_tile) {
    HostScope hs(ctx, "hmm_template");
    const Structure& S = *H.S;
    const Block& R = S.blocks[root];
    auto T = std::make_shared<JobTemplate>();
    // leaves of the subtree, depth-first
    std::vector<int> leaves;
    {
        std::vector<int> stack{root};
        while (!stack.empty()) {
            int b = stack.back();
            stack.pop_back();
            const Block& B = S.blocks[b];
            if (B.kind == KIND_NODE) {
                for (int c = S.q * S.q - 1; c >= 0; --c) stack.push_back(B.first_child + c);
            } else if (B.m > 0 && B.n > 0) {
                leaves.push_back(b);
            }
        }
    }
    // phase 1 items
    std::vector<P1T> p1;
    std::vector<int> p1_box;   // wide: source box of every item
    std::vector<long long> t_rel(leaves.size(), -1);
    long long t_rows = 0;
    for (size_t li = 0; li < leaves.size(); ++li) {
        const int b = leaves[li];
        const Block& B = S.blocks[b];
        if (B.kind != KIND_LOWRANK || H.rank[b] == 0) continue;
        P1T it{};
        if (!trans) {
            it.w = H.V(b) - H.data.get();
            it.nin = B.n;
            it.ldw = B.n;
            it.in_off = B.col_off - R.col_off;
        } else {
            it.w = H.U(b) - H.data.get();
            it.nin = B.m;
            it.ldw = B.m;
            it.in_off = B.row_off - R.row_off;
        }
        it.r = H.rank[b];
        it.t_rel = t_rows;
        t_rel[li] = t_rows;
        t_rows += it.r;
        p1.push_back(it);
        if (row_tile > 32) p1_box.push_back(trans ? B.tgt_box : B.src_box);
    }
    long long c1 = 0;
    int rmax = 0;
    for (P1T& it : p1) {
        it.c0 = c1;
        c1 += it.nin;
        rmax = std::max(rmax, it.r);
    }
    // wide phase-1 tiles: the columns of the W's that share a source box
    // (one input slice), 64 to a tile
    std::vector<W1Source> w1;
    if (row_tile > 32) {
        // by the source box's (offset, size): the few boxes sorted, the items counted in
        std::vector<int> count(S.boxes.size() + 1, 0), boxes;
        for (int b : p1_box)
            if (count[b]++ == 0) boxes.push_back(b);
        std::sort(boxes.begin(), boxes.end(), [&](int a, int b) {
            return std::tie(S.boxes[a].offset, S.boxes[a].count, a) <
                   std::tie(S.boxes[b].offset, S.boxes[b].count, b);
        });
        int at = 0;
        for (int b : boxes) {
            const int n = count[b];
            count[b] = at;
            at += n;
        }
        std::vector<P1T> sorted(p1.size());
        for (size_t i = 0; i < p1.size(); ++i) sorted[count[p1_box[i]]++] = p1[i];
        p1.swap(sorted);
        for (size_t i = 0; i < p1.size();) {
            const long long in_off = p1[i].in_off;
            const int nin = p1[i].nin;
            int rows = 0;   // of the group's last tile
            for (; i < p1.size() && p1[i].in_off == in_off && p1[i].nin == nin; ++i)
                for (int j = 0; j < p1[i].r;) {
                    if (rows % kWideTile == 0) {
                        w1.push_back({in_off, (int)i, j, 0, nin});
                        rows = 0;
                    }
                    const int take = std::min(kWideTile - rows, p1[i].r - j);
                    rows += take;
                    w1.back().rows = rows;
                    j += take;
                }
        }
    }
    // phase 2: bucket the leaves by the output clusters they cover
    const Box& outBox = S.boxes[trans ? R.src_box : R.tgt_box];
    const int outBase = trans ? R.col_off : R.row_off;
    const int c0 = outBox.leaf0, nc = outBox.leaf1 - outBox.leaf0;
    std::vector<int> count(nc + 1, 0);
    for (int b : leaves) {
        const Block& B = S.blocks[b];
        const Box& ob = S.boxes[trans ? B.src_box : B.tgt_box];
        for (int c = ob.leaf0; c < ob.leaf1; ++c) count[c - c0 + 1]++;
    }
    for (int c = 0; c < nc; ++c) count[c + 1] += count[c];
    std::vector<int> bucket(count[nc]);
    {
        std::vector<int> fill(count.begin(), count.end() - 1);
        for (size_t li = 0; li < leaves.size(); ++li) {
            const Block& B = S.blocks[leaves[li]];
            const Box& ob = S.boxes[trans ? B.src_box : B.tgt_box];
            for (int c = ob.leaf0; c < ob.leaf1; ++c) bucket[fill[c - c0]++] = (int)li;
        }
    }
    std::vector<P2T> p2;
    std::vector<P2Entry> ent;
    std::vector<int> zero;
    std::vector<int> ent_block;
    long long c2 = 0;
    for (int c = outBox.leaf0; c < outBox.leaf1; ++c) {
        const Box& cl = S.boxes[S.leaf_box[c]];
        if (cl.count == 0) continue;
        const int e0 = (int)ent.size();
        int cbeg = 0;
        for (int bi = count[c - c0]; bi < count[c - c0 + 1]; ++bi) {
            const int li = bucket[bi];
            const int b = leaves[li];
            const Block& B = S.blocks[b];
            P2Entry e{};
            if (B.kind == KIND_DENSE) {
                if (!trans) {
                    e.a = H.D(b) - H.data.get() + (cl.offset - B.row_off);
                    e.lda = B.m;
                    e.transA = 0;
                    e.inner = B.n;
                    e.b_off = B.col_off - R.col_off;
                } else {
                    e.a = H.D(b) - H.data.get() + (long long)(cl.offset - B.col_off) * B.m;
                    e.lda = B.m;
                    e.transA = 1;
                    e.inner = B.m;
                    e.b_off = B.row_off - R.row_off;
                }
                e.b_from_t = 0;
            } else {
                if (H.rank[b] == 0) continue;
                if (!trans) {
                    e.a = H.U(b) - H.data.get() + (cl.offset - B.row_off);
                    e.lda = B.m;
                } else {
                    e.a = H.V(b) - H.data.get() + (cl.offset - B.col_off);
                    e.lda = B.n;
                }
                e.transA = 0;
                e.inner = H.rank[b];
                e.b_from_t = 1;
                e.b_off = t_rel[li];
                e.ldt = H.rank[b];
            }
            e.cbeg = cbeg;
            cbeg += e.inner;
            ent.push_back(e);
            ent_block.push_back(b);
        }
        const int e1 = (int)ent.size();
        for (int r0 = 0; r0 < cl.count; r0 += row_tile) {
            P2T it{};
            it.out_off = cl.offset - outBase;
            it.r0 = r0;
            it.rows = std::min(row_tile, cl.count - r0);
            it.e0 = e0;
            it.e1 = e1;
            it.c0 = c2;
            it.width = cbeg;
            c2 += cbeg;
            if (cbeg == 0) zero.push_back((int)p2.size());
            p2.push_back(it);
        }
    }
    T->n1 = (int)p1.size();
    T->n2 = (int)p2.size();
    T->t_rows = t_rows;
    T->c1 = c1;
    T->c2 = c2;
    T->rmax = rmax;
    T->p1.upload(p1, ctx.stream);
    T->p2.upload(p2, ctx.stream);
    T->ent.upload(ent, ctx.stream);
    T->hzero = zero;
    T->nw1 = (int)w1.size();
    if (row_tile > 32) {
        // chunk prefixes of the wide kernels (chunks of KC inner indices,
        // none spanning two entries): over the W1 tiles, over the row tiles,
        // then every entry's first chunk within its tile
        std::vector<int> prefix(w1.size() + 1 + p2.size() + 1 + ent.size(), 0);
        int* w1cp = prefix.data();
        int* tcp = w1cp + w1.size() + 1;
        int* ekc = tcp + p2.size() + 1;
        for (size_t i = 0; i < w1.size(); ++i) w1cp[i + 1] = w1cp[i] + ceil_div(w1[i].nin, KC);
        for (size_t t = 0; t < p2.size(); ++t) {
            int k = 0;
            for (int e = p2[t].e0; e < p2[t].e1; ++e) {
                ekc[e] = k;
                k += ceil_div(ent[e].inner, KC);
            }
            tcp[t + 1] = tcp[t] + k;
        }
        T->wc1 = w1cp[w1.size()];
        T->wc2 = tcp[p2.size()];
        T->prefix.upload(prefix, ctx.stream);
        // the tiles' columns and the chunks, made on the device: several times
        // the bytes of the lists they come from (first product of 4 columns with
        // a 128 x 128 operator of rank 4 to 13: 1950 us with lists from the host,
        // 720 us)
        T->w1.allocate(w1.size(), ctx.stream);
        T->chunks.allocate((size_t)(T->wc1 + T->wc2), ctx.stream);
        const size_t tiles = w1.size() + p2.size();
        if (tiles > 0) {
            DeviceBuffer<W1Source> src;
            src.upload(w1, ctx.stream);
            LaunchScope ls(ctx, "hmm_template_expand");
            expand_template_kernel<<<(unsigned)tiles, 64, 0, ctx.stream>>>(
                src.get(), (int)w1.size(), T->p1.get(), T->p2.get(), (int)p2.size(), T->ent.get(),
                T->prefix.get(), T->w1.get(), T->chunks.get());
            HMB_CHECK_LAUNCH();
        }
    }
    T->hp1 = std::move(p1);
    T->hp2 = std::move(p2);
    T->hent = std::move(ent);
    T->hent_block = std::move(ent_block);
    return T;
}

}  // namespace

// The layout group of H in its context (created on first use).
LayoutGroup& layout_group(Context& ctx, const HMatrix& H) {
    if (H.group) return *H.group;
    uint64_t h = 1469598103934665603ULL;
    auto mix = [&](const void* p, size_t n) {
        const unsigned char* c = static_cast<const unsigned char*>(p);
        for (size_t i = 0; i < n; ++i) h = (h ^ c[i]) * 1099511628211ULL;
    };
    const uint64_t id = H.S->id;
    mix(&id, sizeof(id));
    mix(&H.max_rank, sizeof(int));
    mix(H.rank.data(), H.rank.size() * sizeof(int));
    auto& L = ctx.layouts;
    for (size_t i = 0; i < L.size(); ++i) {
        LayoutGroup& g = *L[i];
        if (g.hash == h && g.S->id == id && g.max_rank == H.max_rank && g.rank == H.rank) {
            auto keep = L[i];
            L.erase(L.begin() + (long long)i);
            L.push_back(keep);
            H.group = keep;
            return *keep;
        }
    }
    auto g = std::make_shared<LayoutGroup>();
    g->S = H.S;
    g->max_rank = H.max_rank;
    g->rank = H.rank;
    g->hash = h;
    L.push_back(g);
    if (L.size() > kLayoutGroups) L.erase(L.begin());
    H.group = g;
    return *g;
}

std::shared_ptr<JobTemplate> get_template(Context& ctx, const HMatrix& H, int root, bool trans,
                                          int row_tile) {
    HMB_REQUIRE(row_tile >= 1 && row_tile <= 64, HM_ERR_INTERNAL, "row tile out of range");
    LayoutGroup& G = layout_group(ctx, H);
    auto key = std::make_tuple(root, trans ? 1 : 0, row_tile);
    auto it = G.templates.find(key);
    if (it != G.templates.end()) return it->second;
    auto T = build_template(ctx, H, root, trans, row_tile);
    HMB_REQUIRE((T->n1 == 0 || T->p1.get() || T->w1.get()) &&
                    (T->n2 == 0 || (T->p2.get() && T->ent.get())) && (T->nw1 == 0 || T->w1.get()) &&
                    (T->wc1 + T->wc2 == 0 || T->chunks.get()),
                HM_ERR_INTERNAL, "work lists missing on the device");
    G.templates.emplace(key, T);
    return T;
}

namespace {

// Resident CTAs of a persistent kernel of `threads` threads a CTA.
template <typename K>
int persistent_grid(const Context& ctx, K kernel, int threads, size_t smem = 0) {
    return ctas_per_sm(kernel, threads, smem) * ctx.num_sms;
}

// First item of every warp of the narrow phase-1 kernel for split width GW.
const int* warp_starts1(Context& ctx, JobTemplate& T, long long GW) {
    auto f = T.start1.find(GW);
    if (f != T.start1.end()) return f->second.get();
    std::vector<int> st((size_t)GW);
    int item = 0;
    for (long long w = 0; w < GW; ++w) {
        const long long g = w * T.c1 / GW;
        while (item + 1 < (int)T.hp1.size() && T.hp1[item + 1].c0 <= g) ++item;
        st[(size_t)w] = item;
    }
    DeviceBuffer<int>& d = T.start1[GW];
    d.upload(st, ctx.stream);
    return d.get();
}

// First (tile, entry) of every warp of the narrow phase-2 kernel.
const int2* warp_starts2(Context& ctx, JobTemplate& T, long long GW) {
    auto f = T.start2.find(GW);
    if (f != T.start2.end()) return f->second.get();
    std::vector<int2> st((size_t)GW);
    int tile = 0;
    for (long long w = 0; w < GW; ++w) {
        const long long g = w * T.c2 / GW;
        while (tile + 1 < (int)T.hp2.size() && T.hp2[tile + 1].c0 <= g) ++tile;
        const P2T& it = T.hp2[tile];
        int e = it.e0;
        while (e + 1 < it.e1 && T.hent[e + 1].cbeg <= g - it.c0) ++e;
        st[(size_t)w] = make_int2(tile, e);
    }
    DeviceBuffer<int2>& d = T.start2[GW];
    d.upload(st, ctx.stream);
    return d.get();
}

void launch_narrow(Context& ctx, const JobExec* jobs_d, int nj, const JobExec& job0,
                   long long c1, long long c2, int rmax, JobTemplate* single) {
    cudaStream_t st = ctx.stream;
    if (c1 > 0) {
        const long long g = std::min<long long>(ceil_div(c1, kWarps),
                                                persistent_grid(ctx, p1_stream_kernel, kThreads));
        const long long GW = std::min<long long>(g * kWarps, c1);
        const int* starts = single ? warp_starts1(ctx, *single, GW) : nullptr;
        DeviceBuffer<double> S;
        S.allocate((size_t)(2 * GW * rmax), st);
        LaunchScope ls(ctx, "hmm_lowrank_inner");
        p1_stream_kernel<<<(unsigned)g, kThreads, 0, st>>>(jobs_d, nj, job0, c1, GW, S.get(),
                                                               rmax, starts);
        HMB_CHECK_LAUNCH();
    }
    if (c2 > 0) {
        const long long g = std::min<long long>(ceil_div(c2, kWarps),
                                                persistent_grid(ctx, p2_stream_kernel, kThreads));
        const long long GW = std::min<long long>(g * kWarps, c2);
        const int2* starts = single ? warp_starts2(ctx, *single, GW) : nullptr;
        DeviceBuffer<double> S;
        S.allocate((size_t)(2 * GW * 32), st);
        LaunchScope ls(ctx, "hmm_row_tiles");
        p2_stream_kernel<<<(unsigned)g, kThreads, 0, st>>>(jobs_d, nj, job0, c2, GW, S.get(),
                                                               starts);
        HMB_CHECK_LAUNCH();
    }
}

// Inputs of TF32 products: X (n x k, ld ldx, FP64) -> Xf (n x k, ld n,
// FP32 rounded to TF32), one launch for all distinct inputs (blockIdx.y).
struct InConv {
    const double* src;
    float* dst;
    long long ld, n, total;
};

__global__ void in_tf32_kernel(const InConv* __restrict__ cv) {
    const InConv c = cv[blockIdx.y];
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < c.total;
         e += (long long)gridDim.x * blockDim.x) {
        const long long i = e % c.n, j = e / c.n;
        c.dst[e] = round_tf32(c.src[i + j * c.ld]);
    }
}

// Grids and launches of the FP64 tiles (NT columns a tile).
template <int PHASE, int NT, bool ONE>
int wide64_grid(Context& ctx, long long chunks) {
    allow_smem(wide64_kernel<PHASE, NT, ONE>, Tile64<NT>::smem);
    return (int)std::min<long long>(
        chunks, persistent_grid(ctx, wide64_kernel<PHASE, NT, ONE>, WTHREADS, Tile64<NT>::smem));
}

// f(integral_constant<NT>) for nt = 8, 16, 32 or 64.
template <typename F>
void with_tile_columns(int nt, F f) {
    switch (nt) {
        case 8: f(std::integral_constant<int, 8>{}); break;
        case 16: f(std::integral_constant<int, 16>{}); break;
        case 32: f(std::integral_constant<int, 32>{}); break;
        default: f(std::integral_constant<int, 64>{}); break;
    }
}

void wide64_grids(Context& ctx, int nt, bool one, long long c1, long long c2, int& G1, int& G2) {
    with_tile_columns(nt, [&](auto n) {
        constexpr int NT = decltype(n)::value;
        G1 = one ? wide64_grid<1, NT, true>(ctx, c1) : wide64_grid<1, NT, false>(ctx, c1);
        G2 = one ? wide64_grid<2, NT, true>(ctx, c2) : wide64_grid<2, NT, false>(ctx, c2);
    });
}

void launch_wide64(Context& ctx, int nt, const JobExec* jobs_d, int nj, const JobExec& job0, long long n1,
                   long long n2, int G1, int G2, int ct) {
    with_tile_columns(nt, [&](auto n) {
        constexpr int NT = decltype(n)::value;
        constexpr size_t smem = Tile64<NT>::smem;
        if (n1 > 0 && G1 > 0) {
            LaunchScope ls(ctx, "hmm_lowrank_inner");
            const dim3 grid((unsigned)G1, (unsigned)ct);
            if (jobs_d) wide64_kernel<1, NT, false><<<grid, WTHREADS, smem, ctx.stream>>>(jobs_d, nj, job0, n1, G1);
            else wide64_kernel<1, NT, true><<<grid, WTHREADS, smem, ctx.stream>>>(nullptr, 1, job0, n1, G1);
            HMB_CHECK_LAUNCH();
        }
        if (n2 > 0 && G2 > 0) {
            LaunchScope ls(ctx, "hmm_row_tiles");
            const dim3 grid((unsigned)G2, (unsigned)ct);
            if (jobs_d) wide64_kernel<2, NT, false><<<grid, WTHREADS, smem, ctx.stream>>>(jobs_d, nj, job0, n2, G2);
            else wide64_kernel<2, NT, true><<<grid, WTHREADS, smem, ctx.stream>>>(nullptr, 1, job0, n2, G2);
            HMB_CHECK_LAUNCH();
        }
    });
}

void wide_tf32_grids(Context& ctx, long long c1, long long c2, int& G1, int& G2) {
    constexpr size_t smem = sizeof(WideSmem32);
    allow_smem(wide_tf32_kernel<1>, smem);
    allow_smem(wide_tf32_kernel<2>, smem);
    G1 = (int)std::min<long long>(c1, persistent_grid(ctx, wide_tf32_kernel<1>, WTHREADS, smem));
    G2 = (int)std::min<long long>(c2, persistent_grid(ctx, wide_tf32_kernel<2>, WTHREADS, smem));
}

void launch_wide_tf32(Context& ctx, const JobExec* jobs_d, int nj, const JobExec& job0, long long n1,
                      long long n2, int G1, int G2, int ct) {
    constexpr size_t smem = sizeof(WideSmem32);
    cudaStream_t st = ctx.stream;
    if (n1 > 0 && G1 > 0) {
        LaunchScope ls(ctx, "hmm_lowrank_inner_tf32");
        wide_tf32_kernel<1><<<dim3((unsigned)G1, (unsigned)ct), WTHREADS, smem, st>>>(jobs_d, nj, job0,
                                                                                     n1, G1);
        HMB_CHECK_LAUNCH();
    }
    if (n2 > 0 && G2 > 0) {
        LaunchScope ls(ctx, "hmm_row_tiles_tf32");
        wide_tf32_kernel<2><<<dim3((unsigned)G2, (unsigned)ct), WTHREADS, smem, st>>>(jobs_d, nj, job0,
                                                                                     n2, G2);
        HMB_CHECK_LAUNCH();
    }
}

}  // namespace

int* Context::error_word() {
    if (!errword.get()) {
        errword.allocate(1, stream);
        HMB_CUDA(cudaMemsetAsync(errword.get(), 0, sizeof(int), stream));
    }
    return errword.get();
}

int* Context::numerical_word() {
    if (!numword.get()) {
        numword.allocate(1, stream);
        HMB_CUDA(cudaMemsetAsync(numword.get(), 0, sizeof(int), stream));
    }
    return numword.get();
}

void Context::check_numerical() {
    HMB_CUDA(cudaStreamSynchronize(stream));
    if (errword.get()) {
        int e = 0;
        HMB_CUDA(cudaMemcpy(&e, errword.get(), sizeof(int), cudaMemcpyDeviceToHost));
        if (e) {
            HMB_CUDA(cudaMemset(errword.get(), 0, sizeof(int)));
            throw Error(HM_ERR_TIMEOUT, "a bounded device wait gave up (no progress)");
        }
    }
    if (!numword.get()) return;
    int h = 0;
    HMB_CUDA(cudaMemcpy(&h, numword.get(), sizeof(int), cudaMemcpyDeviceToHost));
    if (h) {
        HMB_CUDA(cudaMemset(numword.get(), 0, sizeof(int)));
        throw Error(HM_ERR_NUMERICAL,
                    "a low-rank rounding met NaN or Inf (non-finite block data entered an "
                    "H*H product)");
    }
}

double* Context::pinned_scalar() {
    if (!pinned) HMB_CUDA(cudaMallocHost((void**)&pinned, sizeof(double)));
    return pinned;
}

double* Context::scratch(int slot, long long n) {
    DeviceBuffer<double>& b = scratch_bufs[slot];
    n = std::max<long long>(n, 2);
    if ((long long)b.size() < n) b.allocate((size_t)(n + n / 4), stream);
    return b.get();
}

int* Context::zeroed_counters(long long n) {
    if (n > counters_cap) {
        const long long cap = std::max<long long>(n, 2 * counters_cap);
        counters.allocate((size_t)cap, stream);
        HMB_CUDA(cudaMemsetAsync(counters.get(), 0, (size_t)cap * sizeof(int), stream));
        counters_cap = cap;
    }
    return counters.get();
}

namespace {

void run_jobs_direct(Context& ctx, const std::vector<MatJob>& jobs, bool tf32);

// The jobs in passes of at most 8 columns (the 8-column tiles).
void run_jobs_split(Context& ctx, const std::vector<MatJob>& jobs, int kmax) {
    for (int c0 = 0; c0 < kmax; c0 += 8) {
        std::vector<MatJob> pass(jobs);
        for (MatJob& J : pass) {
            J.k = std::max(0, std::min(8, J.k - c0));
            if (J.k == 0) continue;
            J.in += (long long)c0 * J.ldin;
            J.out += (long long)c0 * J.ldout;
        }
        run_jobs_direct(ctx, pass, false);
    }
}

}  // namespace

// One pass of the 16-column tiles unless passes of 8 columns are asked for: each
// of the two passes reads every block.  128 x 128 points, rank 16: 105 us
// against 144 (9 columns) and 179 (16); 256 x 256, rank 32: 814 against 1117
// and 1383; 32^3, rank 10: 421 against 561 and 705; 16 x 16, rank 4: 16
// against 25 and 33; the transpose alike.
int fp64_split_for(Context& ctx, const std::vector<MatJob>& jobs) {
    int kmax = 0;
    for (const MatJob& J : jobs) kmax = std::max(kmax, J.k);
    if (kmax <= 8) return 2;
    return kmax <= 16 && ctx.fp64_split == 2 ? 2 : 1;
}

void run_jobs(Context& ctx, const std::vector<MatJob>& jobs, bool tf32) {
    if (jobs.empty()) return;
    int kmax = 0;
    for (const MatJob& J : jobs) kmax = std::max(kmax, J.k);
    if (!tf32 && kmax > 8 && fp64_split_for(ctx, jobs) == 2) run_jobs_split(ctx, jobs, kmax);
    else run_jobs_direct(ctx, jobs, tf32);
}

namespace {

void run_jobs_direct(Context& ctx, const std::vector<MatJob>& jobs, bool tf32) {
    if (jobs.empty()) return;
    cudaStream_t st = ctx.stream;
    std::vector<std::shared_ptr<JobTemplate>> tmpl;
    tmpl.reserve(jobs.size());
    int kmax = 0;
    for (const MatJob& J : jobs) {
        HMB_REQUIRE(J.k >= 0, HM_ERR_ARGUMENT, "negative column count");
        kmax = std::max(kmax, J.k);
    }
    // one vector, one job: stream the blocks (matvec.cu)
    if (!tf32 && jobs.size() == 1 && jobs[0].k == 1 && multiply_vector_streamed(ctx, jobs[0])) return;
    // one column: 32-row tiles, work split evenly over all resident warps;
    // more: tiles of 64 rows on the tensor cores (FP64 at the narrowest tile
    // that takes the columns; TF32 when asked, from 9 columns on).  Streaming
    // kernels on the plain FP64 units took 147 us for 5 columns of the 117 x
    // 101 operator (rank 12), the 8-column tiles take 74; 139 and 90 us for 4
    // columns of the 128 x 128 one, 50 and 15 for 16 x 16 points of rank 4.
    const bool wide = kmax > 1;
    tf32 = tf32 && kmax > 8;
    const int nt = kmax <= 8 ? 8 : kmax <= 16 ? 16 : kmax <= 32 ? 32 : 64;   // FP64 tile columns
    const int row_tile = wide ? 64 : 32;
    for (const MatJob& J : jobs) tmpl.push_back(get_template(ctx, *J.H, J.root, J.trans, row_tile));
    const int ct = ceil_div(std::max(kmax, 1), kWideTile);   // wide column tiles
    long long t_total = 0, c_total = 0;
    std::vector<long long> t_off(jobs.size()), c1_off(jobs.size()), c2_off(jobs.size());
    for (size_t j = 0; j < jobs.size(); ++j) {
        const JobTemplate& T = *tmpl[j];
        t_off[j] = t_total;
        t_total += T.t_rows * jobs[j].k;
        c1_off[j] = c_total;
        c_total += wide ? (long long)T.nw1 * ct : T.n1;
        c2_off[j] = c_total;
        c_total += wide ? (long long)T.n2 * ct : T.n2;
    }
    // wide: persistent grids, 2 partial slots of 64 x 64 per CTA and column tile
    int G1 = 0, G2 = 0;
    long long p_total = 0;
    if (wide) {
        long long c1 = 0, c2 = 0;
        for (size_t j = 0; j < jobs.size(); ++j)
            if (jobs[j].k > 0) {
                c1 += tmpl[j]->wc1;
                c2 += tmpl[j]->wc2;
            }
        if (tf32) wide_tf32_grids(ctx, c1, c2, G1, G2);
        else {
            int live = 0;
            for (const MatJob& J : jobs) live += J.k > 0;
            wide64_grids(ctx, nt, live == 1, c1, c2, G1, G2);
        }
        p_total = 2LL * std::max(G1, G2) * ct * kWideTile * (tf32 ? kWideTile : nt);
    }
    // TF32: the blocks' FP32 copies, the inputs rounded once (inputs shared
    // by several jobs converted once), an FP32 intermediate
    DeviceBuffer<double> tbuf;
    DeviceBuffer<float> tbuf32, inbuf32;
    std::vector<const float*> in32(jobs.size(), nullptr);
    std::vector<int> ldin32(jobs.size(), 0);
    if (tf32) {
        std::map<std::tuple<const double*, int, int, int>, long long> seen;
        std::vector<InConv> conv;
        std::vector<long long> conv_job(jobs.size(), -1), conv_off;
        long long in_total = 0, maxconv = 0;
        for (size_t j = 0; j < jobs.size(); ++j) {
            const MatJob& J = jobs[j];
            if (J.k == 0) continue;
            ensure_tf32_copy(ctx, const_cast<HMatrix&>(*J.H));
            const Block& R = J.H->S->blocks[J.root];
            const int nin = J.trans ? R.m : R.n;
            auto key = std::make_tuple(J.in, J.ldin, nin, J.k);
            auto f = seen.find(key);
            if (f == seen.end()) {
                InConv c{};
                c.src = J.in;
                c.ld = J.ldin;
                c.n = std::max(nin, 1);
                c.total = (long long)nin * J.k;
                f = seen.emplace(key, (long long)conv.size()).first;
                conv.push_back(c);
                conv_off.push_back(in_total);
                in_total += std::max<long long>(c.total, 1);
                maxconv = std::max(maxconv, c.total);
            }
            conv_job[j] = f->second;
            ldin32[j] = std::max(nin, 1);
        }
        inbuf32.allocate((size_t)std::max<long long>(in_total, 1), st);
        tbuf32.allocate((size_t)std::max<long long>(t_total, 1), st);
        for (size_t c = 0; c < conv.size(); ++c) conv[c].dst = inbuf32.get() + conv_off[c];
        for (size_t j = 0; j < jobs.size(); ++j)
            if (conv_job[j] >= 0) in32[j] = conv[(size_t)conv_job[j]].dst;
        HMB_REQUIRE(conv.size() < 65536, HM_ERR_UNSUPPORTED, "too many distinct inputs");
        if (!conv.empty() && maxconv > 0) {
            DeviceBuffer<InConv> dconv;
            dconv.upload(conv, st);
            const long long gx = std::min<long long>(ceil_div(maxconv, 256LL), 2LL * ctx.num_sms);
            LaunchScope ls(ctx, "input_tf32");
            in_tf32_kernel<<<dim3((unsigned)gx, (unsigned)conv.size()), 256, 0, st>>>(dconv.get());
            HMB_CHECK_LAUNCH();
        }
    }
    const long long p_off = tf32 ? 0 : t_total + (t_total & 1);   // the partials on 16 bytes
    tbuf.allocate((size_t)std::max<long long>(p_off + p_total, 1), st);
    int* cnt = ctx.zeroed_counters(std::max<long long>(c_total, 1));
    std::vector<JobExec> ex;
    ex.reserve(jobs.size());
    long long n1 = 0, n2 = 0;
    int rmax = 0;
    size_t first_job = 0;
    for (size_t j = 0; j < jobs.size(); ++j) {
        const MatJob& J = jobs[j];
        if (J.k == 0) continue;
        if (ex.empty()) first_job = j;
        const JobTemplate& T = *tmpl[j];
        JobExec e{};
        e.hb = J.H->data.get();
        e.p1 = T.p1.get();
        e.w1 = T.w1.get();
        e.p2 = T.p2.get();
        e.ent = T.ent.get();
        e.in = J.in;
        e.out = J.out;
        if (tf32) {
            e.hb32 = J.H->data32.get();
            e.in32 = in32[j];
            e.ldin32 = ldin32[j];
            e.T32 = tbuf32.get() + t_off[j];
            e.part = tbuf.get();
        } else {
            e.T = tbuf.get() + t_off[j];
            e.part = tbuf.get() + p_off;
        }
        if (wide) {
            e.w1cp = T.prefix.get();
            e.tcp = e.w1cp + T.nw1 + 1;
            e.ekc = e.tcp + T.n2 + 1;
            e.ch1 = T.chunks.get();
            e.ch2 = e.ch1 + T.wc1;
        }
        e.cnt1 = cnt + c1_off[j];
        e.cnt2 = cnt + c2_off[j];
        e.alpha_scale = J.alpha_scale;
        e.alpha = J.alpha;
        e.beta = J.beta;
        e.ldin = J.ldin;
        e.ldout = J.ldout;
        e.k = J.k;
        e.n1 = wide ? T.nw1 : T.n1;
        e.n2 = T.n2;
        e.ct1 = 1;
        e.ct2 = 1;
        e.p1_begin = n1;
        e.p2_begin = n2;
        n1 += wide ? T.wc1 : T.c1;
        n2 += wide ? T.wc2 : T.c2;
        rmax = std::max(rmax, T.rmax);
        ex.push_back(e);
    }
    if (ex.empty()) return;
    DeviceBuffer<JobExec> dex;
    const JobExec* jobs_d = nullptr;
    if (ex.size() > 1) {
        dex.upload(ex, st);
        jobs_d = dex.get();
    }
    const JobExec job0 = ex[0];
    const int nj = (int)ex.size();
    if (!wide) {
        JobTemplate* single = nj == 1 ? tmpl[first_job].get() : nullptr;
        launch_narrow(ctx, jobs_d, nj, job0, n1, n2, rmax, single);
        launch_zero_tiles(ctx, tmpl, jobs, jobs_d, job0);
        return;
    }
    HMB_REQUIRE(ct < 65536, HM_ERR_UNSUPPORTED, "too many columns");
    if (tf32) launch_wide_tf32(ctx, jobs_d, nj, job0, n1, n2, G1, G2, ct);
    else launch_wide64(ctx, nt, jobs_d, nj, job0, n1, n2, G1, G2, ct);
    // row tiles without entries: output = beta * output
    launch_zero_tiles(ctx, tmpl, jobs, jobs_d, job0);
}

}  // namespace

}  // namespace hmb
