"""H*H products between matrices whose blocks all have ranks of their own (0 to
12, on two levels): the node x low-rank products of one launch then have column
counts from 1 to 12, so its tiles hold columns that some jobs do not have.
maxRank is the blocks' size, so the product is exact: dense algebra, up to 16
roundings of a few 1e-15 a block and the sampled products' orthonormal bases,
below 1e-11."""
import struct

import numpy as np
import pytest

import dmhm_b200 as D
from helpers import relerr
from test_dense_round_edges_gpu import children

pytestmark = pytest.mark.gpu


def mixed_matrix(sizes, levels, maxrank, rng, ranks):
    n = sizes[0] * sizes[1]
    M = np.zeros((n, n))
    out = [struct.pack("=iiii??", levels, maxrank, 0, 0, False, True),
           struct.pack("=iiii", *[s for s in sizes for _ in (0, 1)]), struct.pack("=iiii", 0, 0, 0, 0)]

    def walk(t, s, level):
        m, k = t[2][0] * t[2][1], s[2][0] * s[2][1]
        at = np.s_[t[1]:t[1] + m, s[1]:s[1] + k]
        if max(abs(a - b) for a, b in zip(t[0], s[0])) > 1:
            r = int(rng.integers(ranks[0], ranks[1] + 1))
            U, V = rng.standard_normal((m, r)), rng.standard_normal((k, r))
            M[at] = U @ V.T
            out.append(struct.pack("=ii", 2, r) + U.T.tobytes() + V.T.tobytes())
        elif level < levels - 1:
            out.append(struct.pack("=i", 0))
            for tc in children(t):
                for sc in children(s):
                    walk(tc, sc, level + 1)
        else:
            d = rng.standard_normal((m, k))
            M[at] = d
            out.append(struct.pack("=ii", 3, 0) + np.ascontiguousarray(d.T).tobytes())

    root = ((0, 0), 0, tuple(sizes))
    walk(root, root, 0)
    return b"".join(out) + b"\0" * 4, M


@pytest.mark.parametrize("sizes,ranks", [((32, 32), (0, 12)), ((16, 32), (0, 7)), ((32, 32), (1, 2))])
def test_products_of_mixed_ranks(sizes, ranks):
    rng = np.random.default_rng(sizes[1] + ranks[1])
    c = D.Context(0)
    c.set_oversample(0)          # (samples as many as the block's columns: a full basis)
    (pa, a), (pb, b) = (mixed_matrix(sizes, 4, sizes[0] * sizes[1] // 16, rng, ranks) for _ in range(2))
    A, B = (D.HMat2d.Unpack(p, ctx=c) for p in (pa, pb))
    P = rng.standard_normal((sizes[0] * sizes[1], 3))
    for k in (1, 3, 20):
        X = rng.standard_normal((sizes[0] * sizes[1], k))
        assert relerr(A.Multiply(1.0, X), a @ X) < 1e-13
        assert relerr(A.TransposeMultiply(1.0, X), a.T @ X) < 1e-13
    assert relerr(A.Multiply(-0.5, B).Multiply(1.0, P), -0.5 * a @ (b @ P)) < 1e-11
