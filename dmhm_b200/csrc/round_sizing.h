// Which rounding kernel takes an op, and the shared memory of the register
// form (round_reg.cuh).
#pragma once
#include <algorithm>

#include "lowrank.h"

namespace hmb {

namespace reground {

constexpr int kSlabMax = 64;    // rows of a slab
constexpr int kChunk = 4;       // inner products exchanged per barrier in step 6

// Shared memory of a CTA of NW warps whose ops have at most `cols` columns
// (stacked rank or dense width) and `rout` output columns.  Passed by value and
// addressed from the shared array in every function, so that the accesses stay
// shared-memory ones and the offsets stay in registers.
struct Layout {
    int cp, rp, ld, rows;   // padded columns, output columns; matrix ld, rows
    int part, rowt, chunk, tau, nrm, jex, order, mat, total;
    __host__ __device__ Layout(int nw, int cols, int rout)
        : cp((cols + 31) & ~31), rp((rout + 31) & ~31),
          ld((cols > rp ? cols : rp) | 1), rows((cols + 1) & ~1) {
        part = 2 * nw * kSlabMax;                 // us: 2 x nw x 64
        rowt = part + 3 * nw * cp;                // part: 3 x nw x cp
        tau = rowt + 2 * cp;                      // rowt: 2 x cp
        // the exchange buffers of the sweeps (jex: 2 x nw x 32) and of step 6
        // (chunk: 2 x nw x kChunk x rp) take the place of part and rowt
        chunk = jex = part;
        const int other = part + 2 * nw * (kChunk * rp > 32 ? kChunk * rp : 32);
        if (other > tau) tau = other;
        nrm = tau + cp;
        order = nrm + cp + 2;                     // nrm: cp + 2
        mat = (order + cp + 4 + 1) & ~1;          // order (ints) and one flag
        total = mat + rows * ld + 2;
    }
};

// Rows that nw warps hold for `cols` columns (0: more columns than any slab).
// A lane's share of a slab takes 64 registers at most, so that the broadcast
// reads of a step stay in flight beside it and 16 warps share an SM: twice the
// rows (half the warps) took 14 % longer on 64 x 64 blocks of rank 16 and
// 40 % longer on 72-row complex ones.
__host__ __device__ inline int slab_rows(int cols, int nw, bool fp32) {
    const int rows = cols <= 32 ? 32 : cols <= 64 ? 16 : cols <= 96 ? 12 : 0;
    return nw * (fp32 ? 2 * rows : rows);
}

}  // namespace reground

constexpr int kRegCols = 96;   // most columns of an op of the register form

// Columns of the matrix an op rounds: its stacked rank, or a dense block's width.
inline int op_columns(const RoundOp& op) {
    return op.kind == ROUND_DENSE ? op.n : op.r1 + (op.kind == ROUND_GENERAL ? op.r2 : 0);
}

// Columns an op needs of the register form's layout.  A dense block's update
// U2 V2^T goes through U2^T U_out (r2 rows of the core matrix), and r2 may
// exceed the block's width: a rank above the block size is legal in an
// unpacked matrix, and a product takes it over.
inline int layout_columns(const RoundOp& op) {
    const int c = std::max(op_columns(op), op.rout);
    return op.kind == ROUND_DENSE && op.beta != 0.0 ? std::max(c, op.r2) : c;
}

// Warps the register form (round_reg.cuh) needs to hold an op: 4 or 8; 16 when
// its stacks do not fit (the general kernel runs the worker then).  Small ops
// would fit 1 or 2 warps, but every step waits for the same chain of
// operations whatever its width, and one kernel for all ops of a list shares
// the instruction cache (64 x 64 blocks of rank 16, whole product: 16.0 ms;
// with 1 and 2 warps where they fit 18.8 ms, with 8 warps for all 24 ms).
inline int reg_warps(const RoundOp& op, bool fp32) {
    if (op.kind == ROUND_SET || op.kind == ROUND_CONCAT) return 4;
    const int cols = layout_columns(op);
    if (cols > kRegCols) return 16;
    for (int nw = 4; nw <= 8; nw *= 2)
        if (std::max(std::max(op.m, op.n), cols) <= reground::slab_rows(cols, nw, fp32)) return nw;
    return 16;
}

}  // namespace hmb
