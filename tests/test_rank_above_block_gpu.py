"""Blocks whose stored rank exceeds their size (legal in an unpacked matrix:
any rank >= 0) as the state that a dense x dense compression of an H*H product
adds to, from ranks just above the block to past the register form's columns.
The products are exact (ranks up to the block size are kept), so they agree
with dense algebra to rounding."""
import struct

import numpy as np
import pytest

import dmhm_b200 as D
from helpers import relerr

pytestmark = pytest.mark.gpu
SIDE, LEVELS = 16, 3          # 16 leaf boxes of 16 points


def boxes(level):
    """(coordinates, offset, points) of the boxes of a level, depth first."""
    out = [((0, 0), 0, SIDE * SIDE)]
    for _ in range(level):
        out = [((2 * c[0] + (q & 1), 2 * c[1] + (q >> 1)), o + q * n // 4, n // 4)
               for c, o, n in out for q in range(4)]
    return out


def pack(maxrank, dense, low):
    """Wire format of a matrix with the given leaf blocks: dense[(t, s)] and
    low[(t, s)] = (U, V) by leaf coordinates; absent dense blocks are zero,
    absent low-rank blocks empty."""
    out = [struct.pack("=iiii??", LEVELS, maxrank, 0, 0, False, True),
           struct.pack("=iiii", SIDE, SIDE, SIDE, SIDE), struct.pack("=iiii", 0, 0, 0, 0)]

    def walk(t, s, level):
        if max(abs(a - b) for a, b in zip(t, s)) > 1:
            U, V = low.get((t, s), (np.zeros((0, 0)), np.zeros((0, 0))))
            out.append(struct.pack("=ii", 2, U.shape[1]) + U.T.tobytes() + V.T.tobytes())
        elif level < LEVELS - 1:
            out.append(struct.pack("=i", 0))
            kids = [[(2 * b[0] + (q & 1), 2 * b[1] + (q >> 1)) for q in range(4)] for b in (t, s)]
            for tc in kids[0]:
                for sc in kids[1]:
                    walk(tc, sc, level + 1)
        else:
            d = dense.get((t, s), np.zeros((16, 16)))
            out.append(struct.pack("=ii", 3, 0) + np.ascontiguousarray(d.T).tobytes())

    walk((0, 0), (0, 0), 0)
    return b"".join(out) + b"\0" * 4


def full(dense, low):
    at = {c: o for c, o, _ in boxes(LEVELS - 1)}
    M = np.zeros((SIDE * SIDE, SIDE * SIDE))
    for (t, s), d in dense.items():
        M[at[t]:at[t] + 16, at[s]:at[s] + 16] = d
    for (t, s), (U, V) in low.items():
        M[at[t]:at[t] + 16, at[s]:at[s] + 16] = U @ V.T
    return M


@pytest.mark.parametrize("rank", [17, 20, 33, 64, 96, 97, 130])
@pytest.mark.parametrize("low_precision", [False, True])
def test_dense_compression_onto_a_rank_above_the_block(rank, low_precision):
    rng = np.random.default_rng(rank)
    leaf = [c for c, _, _ in boxes(LEVELS - 1)]
    near = [(t, s) for t in leaf for s in leaf if max(abs(a - b) for a, b in zip(t, s)) <= 1]
    da = {ts: rng.standard_normal((16, 16)) for ts in near}
    db = {ts: rng.standard_normal((16, 16)) for ts in near}
    la = {((2, 0), (0, 0)): (rng.standard_normal((16, rank)), rng.standard_normal((16, rank)))}
    c = D.Context(0)
    c.set_low_precision(low_precision)
    A = D.HMat2d.Unpack(pack(rank, da, la), ctx=c)
    B = D.HMat2d.Unpack(pack(rank, db, {}), ctx=c)
    a, b = full(da, la), full(db, {})
    P = rng.standard_normal((SIDE * SIDE, 4))
    assert relerr(A.Multiply(1.0, P), a @ P) < 1e-13
    # FP64: a few roundings of 1e-15 each; FP32: its sweeps stop at couplings of 1e-6
    tol = 1e-5 if low_precision else 1e-12
    assert relerr(A.Multiply(1.0, B).Multiply(1.0, P), a @ (b @ P)) < tol
    if rank > 64:       # (an update stacks 2 rank columns, 128 at most)
        return
    X = D.HMat2d(ctx=c).CopyFrom(A)
    A.Multiply(0.5, B, -0.7, X)
    assert relerr(X.Multiply(1.0, P), 0.5 * (a @ (b @ P)) - 0.7 * (a @ P)) < tol


@pytest.mark.parametrize("low_precision", [False, True])
def test_dense_compression_that_cancels(low_precision):
    """C + A B where a low-rank block of C nearly cancels the dense x dense
    product added to it: the sum is formed in FP64 before it is rounded, also by
    the FP32 roundings, so what is left (1e-4 of the parts) keeps the
    precision's own error: 1e-5 in FP32 (couplings of 1e-6), 1e-15 / 1e-4 and a
    factor 100 for the sums in FP64."""
    rng = np.random.default_rng(5)
    t, k, s = (2, 0), (1, 0), (0, 0)
    a, b = rng.standard_normal((16, 16)), rng.standard_normal((16, 16))
    rest = 1e-4 * rng.standard_normal((16, 16))
    c = D.Context(0)
    c.set_low_precision(low_precision)
    A = D.HMat2d.Unpack(pack(16, {(t, k): a}, {}), ctx=c)
    B = D.HMat2d.Unpack(pack(16, {(k, s): b}, {}), ctx=c)
    X = D.HMat2d.Unpack(pack(16, {}, {(t, s): (rest - 0.5 * a @ b, np.eye(16))}), ctx=c)
    A.Multiply(0.5, B, 1.0, X)
    got = X.Multiply(1.0, np.eye(SIDE * SIDE))
    at = {q: o for q, o, _ in boxes(LEVELS - 1)}
    assert relerr(got[at[t]:at[t] + 16, at[s]:at[s] + 16], rest) < (1e-5 if low_precision else 1e-9)


@pytest.mark.parametrize("low_precision", [False, True])
@pytest.mark.parametrize("rank", [4, 16, 31])
def test_sampled_products_of_a_small_matrix(rank, low_precision):
    """One low-rank approximation of a product of 256 points (the orthonormal
    form of the register roundings, 8 warps): exact where the product's rank is
    the sample's."""
    rng = np.random.default_rng(rank)
    U, V = rng.standard_normal((16, rank)), rng.standard_normal((16, rank))
    dense = {((1, 1), (2, 1)): U @ V.T}
    b = {((2, 1), (q, 2)): rng.standard_normal((16, 16)) for q in (1, 2, 3)}
    c = D.Context(0)
    c.set_oversample(1)
    c.set_low_precision(low_precision)
    A, B = (D.HMat2d.Unpack(pack(rank, d, {}), ctx=c) for d in (dense, b))
    got_u, got_v = A.LowRankProduct(1.5, B)
    P = rng.standard_normal((SIDE * SIDE, 3))
    assert relerr(got_u @ (got_v.T @ P), 1.5 * full(dense, {}) @ (full(b, {}) @ P)) < (
        1e-5 if low_precision else 1e-12)
