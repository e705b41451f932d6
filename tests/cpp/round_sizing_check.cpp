// Host-side check of the rounding kernels' sizing rule (round_sizing.h): for
// every op that the register form takes, its slabs hold the stacks and the
// layout's core matrix has a row for every column that the kernel writes
// there -- the stacked columns, the output columns, and the columns of U2 when
// a dense block is updated (beta != 0), whose rank may exceed the block.
#include <cstdio>

#include "round_sizing.h"

using namespace hmb;

int main() {
    int fails = 0, taken = 0;
    const int dims[] = {1, 4, 9, 16, 33, 64, 81, 96, 97, 128, 256};
    const int ranks[] = {0, 1, 8, 20, 32, 48, 64, 96, 97, 128, 200};
    for (int kind : {ROUND_GENERAL, ROUND_DENSE, ROUND_ORTHO})
        for (int m : dims)
            for (int n : dims)
                for (int r1 : ranks)
                    for (int r2 : ranks)
                        for (double beta : {0.0, 1.0, -0.5})
                            for (bool fp32 : {false, true}) {
                                RoundOp op{};
                                op.kind = kind;
                                op.m = m;
                                op.n = n;
                                op.r1 = kind == ROUND_DENSE ? 0 : r1;
                                op.r2 = kind == ROUND_ORTHO ? 0 : r2;
                                op.beta = beta;
                                op.rout = std::min(std::min(m, n), 24);
                                const int nw = reg_warps(op, fp32);
                                if (nw > 8) continue;
                                ++taken;
                                int need = std::max(op.rout, kind == ROUND_DENSE ? n : op.r1 + op.r2);
                                if (kind == ROUND_DENSE && beta != 0.0) need = std::max(need, op.r2);
                                const int cols = layout_columns(op);
                                const reground::Layout L(nw, cols, op.rout);
                                const size_t bytes = (size_t)L.total * (fp32 ? 4 : 8);
                                if (L.rows < need || L.ld < need || cols > kRegCols ||
                                    std::max(m, n) > reground::slab_rows(cols, nw, fp32) ||
                                    bytes > 227 * 1024) {
                                    if (++fails < 10)
                                        std::printf("fail kind %d m %d n %d r1 %d r2 %d beta %g fp32 %d: "
                                                    "%d rows for %d columns\n",
                                                    kind, m, n, r1, r2, beta, (int)fp32, L.rows, need);
                                }
                            }
    if (fails || taken < 1000) {
        std::printf("%d failures of %d ops\n", fails, taken);
        return 1;
    }
    std::printf("ok\n");
    return 0;
}
