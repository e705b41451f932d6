"""Timed workloads of the library: H-matrix x dense products, H*H products and
inversions through the public entry points, each with the input a program
holds before the call and a plain 64-bit value of what it returns.

Three kinds of case (key "kind"):

* "apply":   y = H x or H^T x for k columns.  H holds dense leaves and full-rank
             low-rank blocks of random entries and is read from the packed wire
             format.  "on": "device" keeps the operands on the GPU and issues
             the product stream-ordered, as an iterative solver does; "host"
             hands numpy arrays to Multiply.
* "product": C = A B with randomized compression, then C applied to k columns.
             "kernel": A and B are the H-matrices of a smooth kernel with
             random row and column scalings, so that every block is rounded;
             "stencil": A is a sparse grid operator and C = A A under a
             compression tolerance.
* "invert":  the inverse of a grid operator applied to k columns: "schulz"
             (FP64, fixed rank), "mixed" (low-precision early iterations under
             a compression tolerance), "helmholtz" (complex), "direct"
             (recursive Schur complements).

Sizes are grid sides in points; "levels" the tree's levels, "rank" its maxRank.
"""
import ctypes
import functools
import math
import struct

import numpy as np
import torch

import dmhm_b200 as D

_CONTEXTS = {}


def _context(oversample=4, tolerance=0.0):
    """A program makes its context once and keeps it."""
    key = (oversample, tolerance)
    if key not in _CONTEXTS:
        ctx = D.Context(0)
        ctx.set_oversample(oversample)
        ctx.set_compression_tolerance(tolerance)
        _CONTEXTS[key] = ctx
    return _CONTEXTS[key]


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # one vector through a small operator: latency and launches
        {"name": "vector_32", "kind": "apply", "x": 32, "y": 32, "z": 0, "levels": 4, "rank": 8,
         "k": 1, "transpose": False, "on": "device"},
        # one vector through the 128 x 128 operator: the bandwidth-bound step of a Krylov solver
        {"name": "vector_128", "kind": "apply", "x": 128, "y": 128, "z": 0, "levels": 5, "rank": 16,
         "k": 1, "transpose": False, "on": "device"},
        # a few columns of the transpose on an odd grid: block solvers, two-sided norms
        {"name": "few_transposed_odd", "kind": "apply", "x": 117, "y": 101, "z": 0, "levels": 5,
         "rank": 12, "k": 5, "transpose": True, "on": "device"},
        # 64 right-hand sides of the 128 x 128 operator: the library's headline product
        {"name": "block_128", "kind": "apply", "x": 128, "y": 128, "z": 0, "levels": 5, "rank": 16,
         "k": 64, "transpose": False, "on": "device"},
        # a block of columns through an octree of odd sizes
        {"name": "block_3d_odd", "kind": "apply", "x": 30, "y": 25, "z": 27, "levels": 4, "rank": 10,
         "k": 24, "transpose": True, "on": "device"},
        # the largest operator and block
        {"name": "block_200", "kind": "apply", "x": 200, "y": 184, "z": 0, "levels": 5, "rank": 24,
         "k": 128, "transpose": False, "on": "device"},
        # product of two full-rank H-matrices at fixed rank: what each Schulz step does twice
        {"name": "product_64", "kind": "product", "of": "kernel", "x": 64, "y": 64, "z": 0,
         "levels": 4, "rank": 16, "tolerance": 0.0, "k": 16},
        # A A of the seven-point operator under a tolerance
        {"name": "product_3d", "kind": "product", "of": "stencil", "x": 32, "y": 32, "z": 32,
         "levels": 4, "rank": 24, "tolerance": 1e-10, "k": 16},
        # the inverse as a user asks for it: iterate until the stop test passes
        {"name": "schulz_64", "kind": "invert", "how": "schulz", "x": 64, "y": 64, "levels": 4,
         "rank": 16, "k": 16},
        # the same in mixed precision with a tolerance, on a grid that does not halve evenly
        {"name": "schulz_mixed_72", "kind": "invert", "how": "mixed", "x": 72, "y": 68, "levels": 4,
         "rank": 16, "k": 16},
        # complex inverse applied to eight right-hand sides
        {"name": "helmholtz_24", "kind": "invert", "how": "helmholtz", "x": 24, "y": 24, "levels": 3,
         "rank": 12, "k": 8},
        # the non-iterative inverse: a long chain of small products
        {"name": "direct_32", "kind": "invert", "how": "direct", "x": 32, "y": 32, "levels": 4,
         "rank": 8, "k": 16},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["apply", "apply", "apply", "product", "invert"])
    if kind == "apply":
        while True:
            if rng.random() < 0.7:
                x = _log_int(rng, 24, 200)
                y, z = max(20, int(x * rng.uniform(0.7, 1.1))), 0
                levels = max(3, 1 + round(math.log2(max(x, y) / rng.uniform(5, 12))))
            else:
                x = _log_int(rng, 14, 36)
                y, z = x + rng.randint(-2, 2), x + rng.randint(-2, 2)
                levels = 3 if x < 24 else 4
            case = {"kind": "apply", "x": x, "y": y, "z": z, "levels": levels,
                    "rank": rng.randint(4, 24),
                    "k": rng.choice([1, 1, rng.randint(2, 8), _log_int(rng, 9, 128)]),
                    "transpose": rng.random() < 0.4,
                    "on": rng.choice(["device", "device", "host"])}
            if work(case)["bytes"] <= work(listed()[5])["bytes"]:
                return case
    if kind == "product":
        if rng.random() < 0.6:
            x = _log_int(rng, 24, 64)
            return {"kind": "product", "of": "kernel", "x": x, "y": min(64, x + rng.randint(-3, 3)),
                    "z": 0, "levels": 3 if x < 40 else 4, "rank": rng.randint(6, 16),
                    "tolerance": rng.choice([0.0, 0.0, 1e-10]), "k": rng.randint(4, 32)}
        x = _log_int(rng, 16, 32)
        return {"kind": "product", "of": "stencil", "x": x, "y": x - rng.randint(0, 3),
                "z": x - rng.randint(0, 3), "levels": 3 if x < 24 else 4,
                "rank": rng.randint(8, 24), "tolerance": rng.choice([0.0, 1e-10]),
                "k": rng.randint(4, 32)}
    how = rng.choice(["schulz", "mixed", "helmholtz", "direct"])
    hi = {"schulz": 64, "mixed": 72, "helmholtz": 24, "direct": 32}[how]
    x = rng.randint(16 if how in ("helmholtz", "direct") else 32, hi)
    y = min(hi, x + rng.randint(-3, 3))
    rank = {"schulz": rng.randint(14, 18), "mixed": rng.randint(14, 18),
            "helmholtz": rng.randint(10, 12), "direct": rng.randint(6, 12)}[how]
    return {"kind": "invert", "how": how, "x": x, "y": y, "levels": 4 if x >= 48 else 3,
            "rank": rank, "k": rng.randint(4, 24)}


# ---------------------------------------------------------------------------
# Grids, trees and packed matrices
# ---------------------------------------------------------------------------
def _sizes(case):
    return tuple(case[a] for a in "xyz" if case.get(a, 0) > 0)


class _Box:
    """One box of the spatial tree: its grid coordinates at its level, its
    points (natural coordinates in hierarchical order) and its children."""

    def __init__(self, coord, origin, size, level, levels, offset):
        self.coord, self.size, self.offset, self.children = coord, size, offset, []
        self.count = int(np.prod(size))
        if level == levels - 1:
            axes = [np.arange(o, o + s) for o, s in zip(origin, size)]
            grid = np.meshgrid(*axes[::-1], indexing="ij")[::-1]      # first axis fastest
            self.points = np.stack([g.reshape(-1) for g in grid], 1)
            return
        at = offset
        for q in range(1 << len(size)):
            bit = [(q >> a) & 1 for a in range(len(size))]
            low = [s // 2 for s in size]
            child = _Box([2 * c + b for c, b in zip(coord, bit)],
                         [o + (h if b else 0) for o, h, b in zip(origin, low, bit)],
                         [s - h if b else h for s, h, b in zip(size, low, bit)],
                         level + 1, levels, at)
            self.children.append(child)
            at += child.count
        self.points = np.concatenate([c.points for c in self.children])


@functools.lru_cache(maxsize=8)
def _tree(sizes, levels):
    root = _Box([0] * len(sizes), [0] * len(sizes), list(sizes), 0, levels, 0)
    blocks = []       # depth first: ("node" | "low" | "dense", target box, source box)

    def walk(t, s):
        if max(abs(a - b) for a, b in zip(t.coord, s.coord)) > 1:
            blocks.append(("low", t, s))
        elif t.children:
            blocks.append(("node", t, s))
            for tc in t.children:
                for sc in s.children:
                    walk(tc, sc)
        else:
            blocks.append(("dense", t, s))

    walk(root, root)
    return root, blocks


def _random_blocks(case, seed):
    """Every block from one pool of normal draws: (kind, t, s, U, V) with
    columns contiguous, dense blocks in U."""
    rng = np.random.default_rng(seed)
    pool = rng.standard_normal(1 << 21)
    _, blocks = _tree(_sizes(case), case["levels"])
    at = rng.integers(0, 1 << 20, size=2 * len(blocks))
    r = case["rank"]
    for i, (kind, t, s) in enumerate(blocks):
        if kind == "node":
            yield kind, t, s, None, None
        elif kind == "low":
            a, b = at[2 * i], at[2 * i + 1]
            yield kind, t, s, pool[a:a + t.count * r].reshape(r, -1), pool[b:b + s.count * r].reshape(r, -1)
        else:
            a = at[2 * i]
            yield kind, t, s, pool[a:a + t.count * s.count].reshape(s.count, t.count), None


@functools.lru_cache(maxsize=2048)
def _kernel_factors(t_size, s_size, shift, rank, scale):
    """Best rank-r factors of exp(-d) / (1 + d), d = |p - q| / scale, between
    two boxes `shift` apart; dense (rank 0) as it is."""
    def grid(size, origin):
        axes = [np.arange(o, o + n) for o, n in zip(origin, size)]
        g = np.meshgrid(*axes[::-1], indexing="ij")[::-1]
        return np.stack([a.reshape(-1) for a in g], 1).astype(float)

    # the tree's order inside a box is the caller's: points come sorted there
    p, q = grid(t_size, (0,) * len(t_size)), grid(s_size, shift)
    d = np.sqrt(((p[:, None, :] - q[None, :, :]) ** 2).sum(-1)) / scale
    k = np.exp(-d) / (1.0 + d)
    if rank == 0:
        return k, None
    u, w, vt = np.linalg.svd(k, full_matrices=False)
    return np.ascontiguousarray((u[:, :rank] * w[:rank]).T), np.ascontiguousarray(vt[:rank])


def _kernel_blocks(case, seed, which):
    """Blocks of D1 K D2 with random diagonal D1, D2 and a unit diagonal."""
    rng = np.random.default_rng([seed, which])
    sizes = _sizes(case)
    root, blocks = _tree(sizes, case["levels"])
    n = root.count
    left, right = rng.uniform(0.5, 1.5, n), rng.uniform(0.5, 1.5, n)
    scale = max(sizes) / 8.0
    for kind, t, s in blocks:
        if kind == "node":
            yield kind, t, s, None, None
            continue
        to, so = t.points.min(0), s.points.min(0)
        rank = 0 if kind == "dense" else case["rank"]
        a, b = _kernel_factors(tuple(t.size), tuple(s.size), tuple(int(v) for v in so - to), rank, scale)

        def order(box, origin):
            rel, stride = box.points - origin, np.cumprod([1] + list(box.size[:-1]))
            return rel @ stride

        ti, si = order(t, to), order(s, so)
        lt, rs = left[t.offset:t.offset + t.count], right[s.offset:s.offset + s.count]
        if kind == "dense":
            block = 0.1 * (lt[:, None] * a[np.ix_(ti, si)] * rs[None, :])
            if t is s:
                block = block + np.eye(t.count)
            yield kind, t, s, np.ascontiguousarray(block.T), None
        else:
            yield kind, t, s, 0.1 * a[:, ti] * lt, b[:, si] * rs


def _pack(case, blocks):
    """The wire format: header, then the block tree depth first."""
    sizes = _sizes(case)
    out = [struct.pack("=iiii??", case["levels"], case["rank"], 0, 0, False, True)]
    out += [struct.pack("=ii", s, s) for s in sizes] + [struct.pack("=ii", 0, 0)] * len(sizes)
    for kind, t, s, u, v in blocks:
        if kind == "node":
            out.append(struct.pack("=i", 0))
        elif kind == "low":
            out += [struct.pack("=ii", 2, u.shape[0]), u.tobytes(), v.tobytes()]
        else:
            out += [struct.pack("=ii", 3, 0), u.tobytes()]
    out.append(b"\0" * 4)
    return b"".join(out)


def _unpack(case, blocks, ctx):
    cls = D.HMat3d if len(_sizes(case)) == 3 else D.HMat2d
    return cls.Unpack(_pack(case, blocks), ctx=ctx)


def _multiply(blocks, x, transpose=False):
    """H x block by block in numpy."""
    y = np.zeros_like(x)
    for kind, t, s, u, v in blocks:
        if kind == "node":
            continue
        rows, cols = slice(t.offset, t.offset + t.count), slice(s.offset, s.offset + s.count)
        if transpose:
            y[cols] += u @ x[rows] if kind == "dense" else v.T @ (u @ x[rows])
        else:
            y[rows] += u.T @ x[cols] if kind == "dense" else u.T @ (v @ x[cols])
    return y


def _coefficients(case, seed):
    return 1.0 + np.random.default_rng([seed, 5]).random(int(np.prod(_sizes(case))))


def _right_hand_sides(case, seed, n):
    rng = np.random.default_rng([seed, 7])
    b = rng.standard_normal((n, case["k"]))
    if case.get("how") == "helmholtz":
        b = b + 1j * rng.standard_normal((n, case["k"]))
    return b


def _wavenumber(seed):
    return 2.0 + 8.0 * float(np.random.default_rng([seed, 9]).random())


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def prepare(case, seed):
    sizes = _sizes(case)
    n = int(np.prod(sizes))
    state = {"case": case, "seed": seed}
    b = _right_hand_sides(case, seed, n)
    if case["kind"] == "apply":
        state["H"] = _unpack(case, _random_blocks(case, seed), _context())
        if case["on"] == "host":
            state["B"] = np.asfortranarray(b)
        else:     # column-major n x k blocks, as the library takes them
            state["B"] = torch.from_numpy(np.ascontiguousarray(b.T)).cuda()
            state["Y"] = torch.empty_like(state["B"])
        return state
    if case["kind"] == "product":
        ctx = _context(8 if case["of"] == "stencil" else 4, case["tolerance"])
        if case["of"] == "kernel":
            state["A"] = _unpack(case, _kernel_blocks(case, seed, 1), ctx)
            state["M"] = _unpack(case, _kernel_blocks(case, seed, 2), ctx)
        else:
            s = D.operators.stencil(sizes, _coefficients(case, seed), case["levels"])
            state["A"] = D.HMat3d(s, case["levels"], case["rank"], True, *sizes, ctx=ctx)
            state["M"] = state["A"]
    else:
        ctx = _context(4, 1e-10 if case["how"] == "mixed" else 0.0)
        if case["how"] == "helmholtz":
            s = D.operators.helmholtz(sizes, _wavenumber(seed), case["levels"])
        else:
            s = D.operators.stencil(sizes, _coefficients(case, seed), case["levels"])
        state["A"] = D.HMat2d(s, case["levels"], case["rank"], True, *sizes, ctx=ctx)
    state["ctx"] = ctx
    state["B"] = b if case.get("how") == "helmholtz" else torch.from_numpy(b).cuda()
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "apply":
        if case["on"] == "host":
            return (state["H"].TransposeMultiply if case["transpose"] else state["H"].Multiply)(1.0, state["B"])
        b, y = state["B"], state["Y"]
        n = b.shape[1]
        status = D.lib().hm_multiply_dense(
            state["H"].handle, int(case["transpose"]), 1.0, ctypes.c_void_p(b.data_ptr()), n, 0.0,
            ctypes.c_void_p(y.data_ptr()), n, case["k"])
        if status:
            raise RuntimeError(D.lib().hm_last_error().decode())
        return y
    ctx = state["ctx"]
    ctx.set_lcg_states(D.hmat.LCG_SEED, D.hmat.LCG_SEED)    # a reproducible program seeds its draws
    if case["kind"] == "product":
        return state["A"].Multiply(1.0, state["M"]).Multiply(1.0, state["B"])
    x = D.HMat2d(ctx=ctx).CopyFrom(state["A"])
    if case["how"] == "direct":
        x.DirectInvert()
        return x.Multiply(1.0, state["B"])
    if case["how"] == "mixed":
        iterations = x.SchulzInvertMixed(-1, 1.5, 6.0, 1e-8, 0.1)[0]
    else:
        iterations = x.SchulzInvert(-1, 1.5, 6.0, 1e-8)[0]
    return {"x": x.Multiply(1.0, state["B"]), "iterations": iterations}


# ---------------------------------------------------------------------------
# exact / work
# ---------------------------------------------------------------------------
def _grid_operator(case, seed):
    """The operator as (points' hierarchical order, dense matrix or None,
    function applying it), in natural order."""
    sizes = _sizes(case)
    d, n = len(sizes), int(np.prod(sizes))
    natural = np.arange(n)
    stride = np.cumprod([1] + list(sizes[:-1]))
    complex_case = case.get("how") == "helmholtz"
    c = None if complex_case else _coefficients(case, seed)
    if complex_case:
        diag = np.full(n, 2.0 * d + 0.2j - (_wavenumber(seed) / (sizes[0] + 1)) ** 2)
    else:
        diag = 2.0 * d * c + 0.1
    pairs = []
    for a in range(d):
        i = natural[(natural // stride[a]) % sizes[a] < sizes[a] - 1]
        j = i + stride[a]
        pairs.append((i, j, np.full(len(i), -1.0) if complex_case else -np.minimum(c[i], c[j])))
    root, _ = _tree(sizes, case["levels"])
    return root.points @ stride, diag, pairs


def exact(case, seed):
    n = int(np.prod(_sizes(case)))
    b = _right_hand_sides(case, seed, n)
    if case["kind"] == "apply":
        y = _multiply(_random_blocks(case, seed), b, case["transpose"])
        return y if case["on"] == "host" else np.ascontiguousarray(y.T)
    if case["kind"] == "product" and case["of"] == "kernel":
        return _multiply(_kernel_blocks(case, seed, 1), _multiply(_kernel_blocks(case, seed, 2), b))
    order, diag, pairs = _grid_operator(case, seed)
    natural = np.empty_like(b)
    natural[order] = b
    if case["kind"] == "product":
        def operator(v):
            out = diag[:, None] * v
            for i, j, w in pairs:
                out[i] += w[:, None] * v[j]
                out[j] += w[:, None] * v[i]
            return out
        return operator(operator(natural))[order]
    a = np.diag(diag)
    for i, j, w in pairs:
        a[i, j] = w
        a[j, i] = w
    x = torch.linalg.solve(torch.from_numpy(a).cuda(), torch.from_numpy(natural).cuda()).cpu().numpy()[order]
    return x if case["how"] == "direct" else {"x": x, "iterations": None}


def _entries(case):
    """(dense entries, low-rank U and V entries at full rank, rank sum)."""
    _, blocks = _tree(_sizes(case), case["levels"])
    dense = sum(t.count * s.count for kind, t, s in blocks if kind == "dense")
    low = [(t.count + s.count, min(t.count, s.count)) for kind, t, s in blocks if kind == "low"]
    return dense, sum(v * min(case["rank"], w) for v, w in low)


def work(case):
    """An H-matrix product reads every stored entry, the input and writes the
    output: two operations per entry and column.  An H*H product or inverse
    reads its operand and writes its result once; its operations are counted
    as one product of the stored entries with maxRank columns, the least that
    any compression of the result needs (real form for the complex case)."""
    n = int(np.prod(_sizes(case)))
    if case["kind"] == "product" and case["of"] == "stencil":
        # A's admissible blocks are empty, and so are the product's
        _, blocks = _tree(_sizes(case), case["levels"])
        dense, low = sum(t.count * s.count for kind, t, s in blocks if kind == "dense"), 0
    else:
        dense, low = _entries(case)
    entries, k = dense + low, case["k"]
    if case["kind"] == "apply":
        return {"bytes": 8.0 * (entries + 2 * n * k), "flops": 2.0 * entries * k}
    f = 4.0 if case.get("how") == "helmholtz" else 1.0
    moved = 3 if case["kind"] == "product" else 2
    return {"bytes": f * 8.0 * (moved * entries + 2 * n * k),
            "flops": f * 2.0 * entries * (2 * case["rank"] + k)}
