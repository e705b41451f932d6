"""Dense leaf updates and leaf products of an H*H product at the edges of their
64 x 64 tiles: leaves of 4, 16, 25, 64, 76 and 121 points (one to four tiles,
odd leading dimensions), fresh products with real alpha and updates with beta
0, 1 and other, against the oracle's H*H (src/HMat2d/MultiplyHMat-incl.hpp) on
operators whose product is exact at the rank used (the sparse stencil: no
truncation, so products agree to rounding, 1e-12)."""
import numpy as np
import pytest

import dmhm_b200 as D
from helpers import relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes,L", [((8, 8), 3), ((16, 16), 3), ((20, 20), 3), ((32, 32), 3),
                                     ((36, 34), 3), ((44, 44), 3)])
def test_leaf_algebra_edges(sizes, L):
    ops = D.operators
    c = D.Context(0)
    c.set_oversample(0)
    N = sizes[0] * sizes[1]
    r = min(2 * max(sizes) // 4, (sizes[0] // 4) * (sizes[1] // 4))
    S = [ops.stencil(sizes, ops.uniform_coefficients(sizes, s), L) for s in (1, 2, 3)]
    A, B, Cm = (D.HMat2d(s, L, r, True, *sizes, ctx=c) for s in S)
    a, b, cc = (ops.dense_from_sparse(s) for s in S)
    P = np.random.default_rng(3).standard_normal((N, 5))
    AB = a @ (b @ P)
    got = A.Multiply(-0.75, B)
    assert relerr(got.Multiply(1.0, P), -0.75 * AB) < 1e-12
    for beta in (0.0, 1.0, -2.0):
        X = D.HMat2d(ctx=c).CopyFrom(Cm)
        A.Multiply(0.5, B, beta, X)
        assert relerr(X.Multiply(1.0, P), 0.5 * AB + beta * (cc @ P)) < 1e-12
