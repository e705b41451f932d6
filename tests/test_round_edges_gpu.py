"""Low-rank roundings at the edges of the register form, in FP64 and in the FP32
form of the low-precision phase: one, two and three columns a lane (32 | 34, 64
| 66, 96 | 98 stacked columns), every slab height (8 to 32 rows in FP64, 64 in
FP32), 4 and 8 warps, the sweeps from shared memory (65 to 96 columns) and the
general kernel beyond.

Each block of an update is compared with the best approximation of the same
rank by LAPACK's SVD: the error may exceed the best one by rounding only.  FP64:
a rounding of the stack's size m + n + k times 2.2e-16, below 1e-13 of the
block.  FP32: its sweeps stop at couplings of 1e-6, below 1e-5."""
import numpy as np
import pytest

import dmhm_b200 as D

pytestmark = pytest.mark.gpu

# grid (all with 3 levels: 16 leaves), rank; 2 rank columns on leaves of m rows
CASES = [((12, 12), 3), ((20, 20), 16), ((32, 32), 16), ((32, 32), 17), ((36, 36), 30),
         ((36, 36), 32), ((36, 36), 33), ((36, 36), 40), ((36, 36), 47), ((36, 36), 48),
         ((36, 36), 49), ((44, 44), 15), ((44, 44), 40), ((48, 48), 20), ((64, 64), 8),
         ((68, 68), 8)]


@pytest.mark.parametrize("low_precision", [False, True])
@pytest.mark.parametrize("sizes,r", CASES)
def test_updates_are_best_approximations(sizes, r, low_precision):
    from oracle import dmhm_oracle as O
    c = D.Context(0)
    c.set_low_precision(low_precision)
    coef = D.operators.uniform_coefficients(sizes, 1)
    S = D.operators.stencil(sizes, coef, 3)
    A, B = (D.HMat2d(S, 3, r, True, *sizes, ctx=c) for _ in range(2))
    A.SetToRandom()
    B.SetToRandom()
    rng = O.Rng()
    Ao, Bo = (O.build_stencil_hmat(2, sizes, 3, r, coef) for _ in range(2))
    O.set_to_random(Ao, rng)
    O.set_to_random(Bo, rng)
    A.UpdateWith(-0.7, B)
    got = A.Multiply(1.0, np.eye(A.Height()))
    eps = 1e-5 if low_precision else 1e-13
    seen = 0
    for a, b in zip(Ao.leaves(), Bo.leaves()):
        if a.kind == O.DENSE:
            continue
        M = a.U @ a.V.T - 0.7 * b.U @ b.V.T
        s = np.linalg.svd(M, compute_uv=False)
        X = got[a.tgt_off:a.tgt_off + M.shape[0], a.src_off:a.src_off + M.shape[1]]
        best, norm = np.linalg.norm(s[r:]), np.linalg.norm(s)
        # errors of the kept part and of the cut add in squares: (best^2 + e^2)^(1/2)
        assert np.linalg.norm(X - M) <= np.hypot(best, eps * norm) + eps * best
        assert np.linalg.svd(X, compute_uv=False)[r:].max(initial=0.0) < 1e-12 * norm
        seen += 1
        if seen == 24:      # (blocks of a list differ in their content only)
            break
    assert seen == 24
