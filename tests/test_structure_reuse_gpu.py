"""Matrices of one topology and equal ranks on grids of different sizes, one
after the other on one context, each freed before the next is made (so that its
block structure may lie where the last one lay): products must come from lists
of their own sizes.  Against dense algebra of the sparse operator, whose product
with itself is exact at the rank used."""
import numpy as np
import pytest

import dmhm_b200 as D
from helpers import relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("levels", [2, 3])
def test_products_after_a_matrix_of_the_same_topology(levels):
    ops = D.operators
    c = D.Context(0)
    c.set_oversample(4)
    rng = np.random.default_rng(levels)
    for side in (8, 16, 12, 20, 8, 24, 16):
        sizes = (side, side)
        S = ops.stencil(sizes, ops.uniform_coefficients(sizes, side), levels)
        a = ops.dense_from_sparse(S)
        H = D.HMat2d(S, levels, 16, True, *sizes, ctx=c)
        for k in (1, 4, 12, 64):
            X = rng.standard_normal((side * side, k))
            assert relerr(H.Multiply(1.0, X), a @ X) < 1e-13, (side, k)
            assert relerr(H.TransposeMultiply(1.0, X), a.T @ X) < 1e-13, (side, k)
        assert relerr(H.Multiply(1.0, H).Multiply(1.0, X), a @ (a @ X)) < 1e-12, side
        del H, S
