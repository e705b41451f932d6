"""One column through the general lists (the streaming kernels that take it where
the block-streamed plan does not: leaves of more than 512 points, ranks above
128, several products in one launch), against dense algebra."""
import numpy as np
import pytest

import dmhm_b200 as D
from helpers import relerr
from test_mixed_ranks_gpu import mixed_matrix
from test_rank_above_block_gpu import boxes, full, pack

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(60, 60), (47, 51)])
def test_leaves_beyond_the_streamed_plan(sizes):
    ops = D.operators
    c = D.Context(0)
    S = ops.stencil(sizes, ops.uniform_coefficients(sizes, 3), 2)
    H, a = D.HMat2d(S, 2, 4, True, *sizes, ctx=c), ops.dense_from_sparse(S)
    x = np.random.default_rng(1).standard_normal(sizes[0] * sizes[1])
    for _ in range(2):      # (counters are reused)
        assert relerr(H.Multiply(-2.0, x), -2.0 * (a @ x)) < 1e-13
        assert relerr(H.TransposeMultiply(1.0, x), a.T @ x) < 1e-13


def test_ranks_beyond_the_streamed_plan():
    rng = np.random.default_rng(2)
    leaf = [c for c, _, _ in boxes(2)]
    dense = {(t, t): rng.standard_normal((16, 16)) for t in leaf[:-1]}     # one row tile is empty
    low = {((3, 3), (0, 0)): (rng.standard_normal((16, 130)), rng.standard_normal((16, 130))),
           ((0, 2), (2, 0)): (rng.standard_normal((16, 5)), rng.standard_normal((16, 5)))}
    c = D.Context(0)
    H, a = D.HMat2d.Unpack(pack(4, dense, low), ctx=c), full(dense, low)
    x = rng.standard_normal(256)
    assert relerr(H.Multiply(1.0, x), a @ x) < 1e-13
    assert relerr(H.TransposeMultiply(3.0, x), 3.0 * (a.T @ x)) < 1e-13


def test_products_of_rank_one_blocks():
    """Node x low-rank products of one column each in one launch; exact up to the
    roundings of a block's products (1e-11, as for other ranks)."""
    rng = np.random.default_rng(3)
    c = D.Context(0)
    c.set_oversample(0)
    (pa, a), (pb, b) = (mixed_matrix((32, 32), 4, 64, rng, (1, 1)) for _ in range(2))
    A, B = (D.HMat2d.Unpack(p, ctx=c) for p in (pa, pb))
    P = rng.standard_normal((1024, 3))
    assert relerr(A.Multiply(1.0, B).Multiply(1.0, P), a @ (b @ P)) < 1e-11
