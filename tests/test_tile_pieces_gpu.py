"""FP64 tiles cut between CTAs, whose partial sums the last piece adds: few
points, so that every tile is cut (one chunk a CTA), with row tiles of 16 of 64
rows, every tile width and one column more, one low-rank block of odd rank (an
odd number of intermediate values in front of the partials), alpha and beta, and
several products on one context (the counters are reused); against dense
algebra to the H x dense tolerance."""
import ctypes as C

import numpy as np
import pytest

import dmhm_b200 as D
from dmhm_b200 import _lib
from helpers import relerr
from test_rank_above_block_gpu import boxes, full, pack

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rank", [0, 3])
@pytest.mark.parametrize("k", [2, 3, 8, 9, 16, 17, 31, 32, 33, 63, 65, 129])
def test_cut_tiles(rank, k):
    import torch
    rng = np.random.default_rng(10 * k + rank)
    leaf = [c for c, _, _ in boxes(2)]
    near = [(t, s) for t in leaf for s in leaf if max(abs(a - b) for a, b in zip(t, s)) <= 1]
    dense = {ts: rng.standard_normal((16, 16)) for ts in near}
    low = {((3, 1), (0, 2)): (rng.standard_normal((16, rank)), rng.standard_normal((16, rank)))}
    c = D.Context(0)
    H, h = D.HMat2d.Unpack(pack(4, dense, low), ctx=c), full(dense, low)
    n = h.shape[0]
    for op, a in ((0, h), (1, h.T), (0, h)):
        X, Y = rng.standard_normal((n, k)), rng.standard_normal((n, k))
        x, y = (torch.tensor(v.T.copy(), device="cuda") for v in (X, Y))
        torch.cuda.synchronize()
        _lib.check(_lib.lib().hm_multiply_dense(H.handle, op, 0.75, C.c_void_p(x.data_ptr()), n, -2.0,
                                                C.c_void_p(y.data_ptr()), n, k))
        c.synchronize()
        assert relerr(y.cpu().numpy().T, 0.75 * (a @ X) - 2.0 * Y) < 1e-13
