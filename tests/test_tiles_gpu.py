"""H x dense in FP64 at the edges of the 64-row tensor-core tiles: every tile
width (8, 16, 32, 64 columns and one more), blocks of odd rank and odd height
(unaligned columns), two row tiles a cluster, the transpose, operands at odd
leading dimensions and off a 16-byte boundary, alpha and beta; against the
oracle's recursive product (src/HMat2d/MultiplyDense-incl.hpp:12-150) to the
H x dense tolerance."""
import ctypes as C

import numpy as np
import pytest

import dmhm_b200 as D
from dmhm_b200 import _lib
from helpers import relerr

pytestmark = pytest.mark.gpu
TOL = 1e-13


@pytest.mark.parametrize("sizes,L,r", [((24, 20), 3, 5), ((36, 36), 3, 7), ((32, 32), 4, 8)])
@pytest.mark.parametrize("k", [2, 7, 8, 9, 16, 17, 32, 33, 41, 64, 65])
def test_tile_edges(sizes, L, r, k):
    import torch
    from oracle import dmhm_oracle as O
    c = D.Context(0)
    coef = D.operators.uniform_coefficients(sizes, 4)
    H = D.HMat2d(D.operators.stencil(sizes, coef, L), L, r, True, *sizes, ctx=c)
    H.SetToRandom()
    Ho = O.build_stencil_hmat(2, sizes, L, r, coef)
    O.set_to_random(Ho, O.Rng())
    N = sizes[0] * sizes[1]
    rng = np.random.default_rng(k)
    X = rng.standard_normal((N, k))
    Y0 = rng.standard_normal((N, k))
    for op, ref in ((0, O.multiply_dense), (1, O.transpose_multiply_dense)):
        for off, pad in ((0, 0), (1, 1), (1, 2)):
            ld = N + pad
            x = torch.zeros(k * ld + off, dtype=torch.float64, device="cuda")
            y = torch.zeros_like(x)
            xv = x[off:].view(k, ld)[:, :N]
            yv = y[off:].view(k, ld)[:, :N]
            xv.copy_(torch.tensor(X.T.copy()))
            yv.copy_(torch.tensor(Y0.T.copy()))
            torch.cuda.synchronize()
            _lib.check(_lib.lib().hm_multiply_dense(
                H.handle, op, -0.5, C.c_void_p(x.data_ptr() + 8 * off), ld, 2.0,
                C.c_void_p(y.data_ptr() + 8 * off), ld, k))
            c.synchronize()
            assert relerr(yv.cpu().numpy().T, -0.5 * ref(Ho, 1.0, X) + 2.0 * Y0) < TOL
