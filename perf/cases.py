"""What a user of this framework has it do, as cases that can be timed and checked.

A case is a dict of plain values: a path through the public entry points and
the matrices that go through it.

    product  resident tiles:   spgemm -> tiled_to_csr (device CSR)
    chain    new matrices:     csr_to_tiled -> spgemm -> tiled_to_csr
    host     host CSR to host CSR in one call (spgemm_csr_host_overlap)
    batch    uneven products kept as one Batch: run, sync, tiled_to_csr of each
    order    order + permute_csr of a matrix that arrives in random order

Matrices are those of the benchmark and the tests (27-point and 5-point
stencils, R-MAT graphs, bands, uniformly random rows), made on the GPU; FP64
values, 32-bit indices, the only types there are.  The seed gives the values
and, where that keeps the number of entries of C, the places too (rows of A
and columns of B of random operands, the arriving order of a grid matrix).
"""
from __future__ import annotations

import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = Path(__file__).resolve().parents[1] / "rw-spgemm_b200"


def _package():
    name = "rw_spgemm_b200"
    if name not in sys.modules:
        spec = importlib.util.spec_from_file_location(name, _PKG / "__init__.py",
                                                      submodule_search_locations=[str(_PKG)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


_ctx = None


def _context():
    """The context a user's program keeps, on torch's current stream."""
    global _ctx
    if _ctx is None:
        _ctx = _package().Context(0)
    return _ctx


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # one small solve step of an application: latency and launches count
        dict(name="small rectangular", path="product", kind="random", m=1500, k=1100, n=1300, lam=8.0),
        # a coarse grid of a multigrid hierarchy, n not a multiple of 16
        dict(name="stencil 21^3", path="product", kind="stencil", nx=21),
        # the benchmark's headline product: a fine 3-D grid, resident in HBM
        dict(name="stencil 64^3", path="product", kind="stencil", nx=64),
        # a 2-D operator assembled anew: conversion, product, result as CSR
        dict(name="laplacian 256^2 chain", path="chain", kind="laplacian", nx=256),
        # very sparse unstructured operands: C has more tiles than A has entries
        dict(name="random 65536", path="product", kind="random", m=65536, k=65536, n=65536, lam=8.0),
        # band times band: dense C tiles
        dict(name="banded 16384", path="product", kind="banded", n=16384, ha=40, hb=40),
        # a band applied to an unstructured matrix
        dict(name="band times random 8192", path="product", kind="mixed", n=8192, ha=32, lam=8.0),
        # graph work (paths of length two): skewed rows, the middle of the served mix ...
        dict(name="rmat 14 A*A^T", path="product", kind="rmat", scale=14, ef=16, aat=True),
        # ... and the largest product here
        dict(name="rmat 16 A*A", path="product", kind="rmat", scale=16, ef=16, aat=False),
        # a program that holds its matrices in host memory
        dict(name="host stencil 48^3", path="host", kind="stencil", nx=48, pinned=True),
        # many uneven products at once, as the server and the autotuner run them
        dict(name="batch of 16", path="batch", count=16, n_min=1024, n_max=16384, spec=0),
        # a grid matrix in random order brought to a narrow band
        dict(name="rcm stencil 40^3", path="order", kind="stencil", nx=40, ordering="rcm"),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _draw_operands(rng, top):
    """Operands of one product; top in (0, 1] scales the largest sizes."""
    kind = rng.choice(["stencil", "laplacian", "random", "random", "banded", "mixed", "rmat"])
    if kind == "stencil":
        return dict(kind=kind, nx=_log(rng, 8, max(12, int(64 * top))))
    if kind == "laplacian":
        return dict(kind=kind, nx=_log(rng, 24, max(48, int(512 * top))))
    if kind == "random":
        hi = max(2048, int(65536 * top))
        n = _log(rng, 800, hi)
        if rng.random() < 0.5:  # square
            return dict(kind=kind, m=n, k=n, n=n, lam=round(rng.uniform(3.0, 10.0), 2))
        return dict(kind=kind, m=n, k=_log(rng, 800, hi), n=_log(rng, 800, hi), lam=round(rng.uniform(3.0, 10.0), 2))
    if kind == "banded":
        return dict(kind=kind, n=_log(rng, 1024, max(4096, int(65536 * top))), ha=rng.randint(8, 64),
                    hb=rng.randint(8, 64))
    if kind == "mixed":
        return dict(kind=kind, n=_log(rng, 1024, max(4096, int(32768 * top))), ha=rng.randint(8, 64),
                    lam=round(rng.uniform(3.0, 10.0), 2))
    return dict(kind=kind, scale=rng.randint(10, 16 if top == 1 else 14), ef=rng.randint(4, 15),
                aat=rng.random() < 0.5)


def draw(rng):
    path = rng.choice(["product"] * 6 + ["chain"] * 2 + ["host", "batch", "order"])
    if path == "batch":
        return dict(path=path, count=rng.randint(3, 16), n_min=1024, n_max=_log(rng, 4096, 16384),
                    spec=rng.randint(1, 1 << 30))
    if path == "order":
        return dict(path=path, kind="stencil", nx=rng.randint(12, 40), ordering=rng.choice(["rcm", "rcm", "degree"]))
    if path == "host":
        return dict(path=path, pinned=rng.random() < 0.5, **_draw_operands(rng, 0.5))
    return dict(path=path, **_draw_operands(rng, 1 if path == "product" else 0.75))


# ---------------------------------------------------------------------------
# matrices (m, n, rowptr, colidx, val) on the device, rows sorted, no duplicates
# ---------------------------------------------------------------------------
def _device():
    return torch.device("cuda", 0) if torch.cuda.is_available() else torch.device("cpu")


def _generator(seed):
    g = torch.Generator(device=_device())
    g.manual_seed(int(seed))
    return g


def _from_keys(m, n, keys, g, lo=-1.0, hi=1.0):
    """CSR of the distinct keys row * n + col."""
    keys = torch.unique(keys)  # sorted
    rows = torch.div(keys, max(n, 1), rounding_mode="floor")
    cols = (keys - rows * n).to(torch.int32)
    rp = torch.zeros(m + 1, dtype=torch.int64, device=keys.device)
    rp[1:] = torch.cumsum(torch.bincount(rows, minlength=m), 0)
    val = torch.rand(keys.numel(), dtype=torch.float64, device=keys.device, generator=g) * (hi - lo) + lo
    return m, n, rp.to(torch.int32), cols, val


def _grid(nx, dims, reach, seed, lo, hi, permute=False):
    """Stencil on an nx^dims grid: all offsets within `reach` (27 points in
    3-D), or the axis neighbours alone (reach 0: 5 points in 2-D)."""
    n = nx ** dims
    dev = _device()
    idx = torch.arange(n, dtype=torch.int64, device=dev)
    axes = [torch.div(idx, nx ** d, rounding_mode="floor") % nx for d in range(dims)]
    steps = [[]]
    for _ in range(dims):
        steps = [s + [o] for s in steps for o in (-1, 0, 1)]
    if not reach:
        steps = [s for s in steps if sum(map(abs, s)) <= 1]
    g = _generator(seed)
    new = torch.randperm(n, device=dev, generator=g) if permute else idx
    keys = []
    for s in steps:
        ok = torch.ones(n, dtype=torch.bool, device=dev)
        to = idx.clone()
        for d, o in enumerate(s):
            ok &= (axes[d] + o >= 0) & (axes[d] + o < nx)
            to += o * nx ** d
        keys.append(new[idx[ok]] * n + new[to[ok]])
    return _from_keys(n, n, torch.cat(keys), g, lo, hi)


def _random(m, n, lam, spec, seed, shuffle):
    """Each row draws Poisson(lam) uniform columns (duplicates merged), one
    pattern for each spec; its rows ("rows") or columns ("cols") then come in
    an order of the seed's, which leaves every product's count as it is."""
    g = _generator(spec)
    per = torch.poisson(torch.full((m,), float(lam), device=_device()), generator=g).to(torch.int64)
    rows = torch.repeat_interleave(torch.arange(m, device=_device()), per)
    cols = torch.randint(0, n, (rows.numel(),), device=_device(), generator=g)
    g = _generator(seed)
    if shuffle == "rows":
        rows = torch.randperm(m, device=_device(), generator=g)[rows]
    else:
        cols = torch.randperm(n, device=_device(), generator=g)[cols]
    return _from_keys(m, n, rows * n + cols, g)


def _banded(n, half, seed):
    g = _generator(seed)
    i = torch.arange(n, dtype=torch.int64, device=_device())[:, None]
    j = i + torch.arange(-half, half + 1, dtype=torch.int64, device=_device())[None, :]
    keys = (i * n + j)[(j >= 0) & (j < n)]
    return _from_keys(n, n, keys, g)


def _rmat(scale, ef, seed):
    """R-MAT graph (0.57, 0.19, 0.19, 0.05), duplicates merged."""
    n = 1 << scale
    g = _generator(100 * scale + ef)
    rows = torch.zeros(ef * n, dtype=torch.int64, device=_device())
    cols = torch.zeros_like(rows)
    for level in range(scale):
        u = torch.rand(rows.numel(), device=_device(), generator=g)
        bit = 1 << (scale - 1 - level)
        rows += (u >= 0.76) * bit
        cols += (((u >= 0.57) & (u < 0.76)) | (u >= 0.95)) * bit
    return _from_keys(n, n, rows * n + cols, _generator(seed))


def _transpose(mat):
    m, n, rp, ci, v = mat
    rows = torch.repeat_interleave(torch.arange(m, device=rp.device), (rp[1:] - rp[:-1]).to(torch.int64))
    keys, at = torch.sort(ci.to(torch.int64) * m + rows)
    rpT = torch.zeros(n + 1, dtype=torch.int64, device=rp.device)
    rpT[1:] = torch.cumsum(torch.bincount(ci, minlength=n), 0)
    return n, m, rpT.to(torch.int32), (keys % m).to(torch.int32), v[at].contiguous()


def _operands(case, seed):
    """[(A, B)] of the case; B is A itself for A*A."""
    if case["path"] == "batch":
        # the sizes and kinds of the products are the case's, the numbers the seed's
        rs = np.random.default_rng(case["spec"])
        out = []
        for p in range(case["count"]):
            n = int(round(math.exp(rs.uniform(math.log(case["n_min"]), math.log(case["n_max"])))))
            pair = []
            for side in range(2):
                s = 1000 * seed + 2 * p + side
                half = int(rs.integers(8, 65))
                pair.append(_banded(n, half, s) if rs.random() < 0.5
                            else _random(n, n, 8.0, n + side, s, ("rows", "cols")[side]))
            out.append(tuple(pair))
        return out
    kind = case["kind"]
    if kind == "stencil":
        A = _grid(case["nx"], 3, 1, seed, 0.5, 1.5, permute=case["path"] == "order")
        return [(A, A)]
    if kind == "laplacian":
        A = _grid(case["nx"], 2, 0, seed, 0.5, 1.5)
        return [(A, A)]
    if kind == "random":
        return [(_random(case["m"], case["k"], case["lam"], 1, 2 * seed, "rows"),
                 _random(case["k"], case["n"], case["lam"], 2, 2 * seed + 1, "cols"))]
    if kind == "banded":
        return [(_banded(case["n"], case["ha"], 2 * seed), _banded(case["n"], case["hb"], 2 * seed + 1))]
    if kind == "mixed":
        return [(_banded(case["n"], case["ha"], 2 * seed), _random(case["n"], case["n"], case["lam"], 2, 2 * seed + 1, "cols"))]
    A = _rmat(case["scale"], case["ef"], seed)
    return [(A, _transpose(A) if case["aat"] else A)]


# ---------------------------------------------------------------------------
# passes
# ---------------------------------------------------------------------------
def _host(t, pinned):
    t = t.cpu()
    return (t.pin_memory() if pinned else t).numpy()


def prepare(case, seed):
    pkg, ctx = _package(), _context()
    pairs = _operands(case, seed)
    st = dict(path=case["path"], ctx=ctx)
    if case["path"] in ("order", "chain"):
        st["A"], st["B"] = pairs[0]
        st["ordering"] = case.get("ordering")
        return st
    if case["path"] == "host":
        (A, B), pin = pairs[0], case["pinned"]
        st["A"] = tuple(x if isinstance(x, int) else _host(x, pin) for x in A)
        st["B"] = None if B is A else tuple(x if isinstance(x, int) else _host(x, pin) for x in B)
        st["out"] = pkg.HostResultBuffers(A[0], _sizes(pairs)[2] + 1)  # the buffers a user's loop keeps
        return st

    def tiles(M):
        return pkg.csr_to_tiled(ctx, *M, pkg.TSG_TILED_CSC_VIEW)

    tiled = []
    for A, B in pairs:
        tA = tiles(A)
        tiled.append((tA, tA if B is A else tiles(B)))
    if case["path"] == "batch":
        st["batch"] = pkg.Batch(ctx, tiled)
    else:
        st["A"], st["B"] = tiled[0]
    return st


def run(state):
    pkg, ctx, path = _package(), state["ctx"], state["path"]
    if path == "product":
        C, _ = pkg.spgemm(ctx, state["A"], state["B"])
        return pkg.tiled_to_csr(ctx, C)
    if path == "chain":
        A = pkg.csr_to_tiled(ctx, *state["A"], pkg.TSG_TILED_CSC_VIEW)
        B = A if state["B"] is state["A"] else pkg.csr_to_tiled(ctx, *state["B"], pkg.TSG_TILED_CSC_VIEW)
        C, _ = pkg.spgemm(ctx, A, B)
        return pkg.tiled_to_csr(ctx, C)
    if path == "host":
        C, _ = pkg.spgemm_csr_host_overlap(ctx, state["A"], state["B"], state["out"])
        return C[2:]
    if path == "batch":
        batch = state["batch"]
        batch.run()
        batch.sync()
        return [pkg.tiled_to_csr(ctx, batch.product(p)) for p in range(batch.count)]
    m, n, rp, ci, v = state["A"]
    old = pkg.order(ctx, state["ordering"], m, n, rp, ci)
    new = torch.empty_like(old)
    new[old.long()] = torch.arange(m, dtype=torch.int32, device=old.device)
    return (old,) + tuple(pkg.permute_csr(ctx, m, n, rp, ci, v, old, new))


# ---------------------------------------------------------------------------
# what a pass cannot do without, and what it should give
# ---------------------------------------------------------------------------
_CHUNK = 1 << 25  # products expanded at a time


def _expand(A, B):
    """Yields (first row, last row, sorted keys row * n + col, values) of the
    products of A's rows, a run of rows at a time, in A's entry order."""
    m, _, rpA, ciA, vA = A
    _, n, rpB, ciB, vB = B
    rpA, rpB = rpA.to(torch.int64), rpB.to(torch.int64)
    lens = (rpB[1:] - rpB[:-1])[ciA.long()]
    upto = torch.zeros(ciA.numel() + 1, dtype=torch.int64, device=lens.device)
    upto[1:] = torch.cumsum(lens, 0)
    at_row = upto[rpA].cpu().numpy()  # products before each row
    r0 = 0
    while r0 < m:
        r1 = max(r0 + 1, int(np.searchsorted(at_row, at_row[r0] + _CHUNK, side="right")) - 1)
        e0, e1 = int(rpA[r0]), int(rpA[r1])
        ln = lens[e0:e1]
        ent = torch.repeat_interleave(torch.arange(e0, e1, device=ln.device), ln)
        at = rpB[ciA[ent].long()] + torch.arange(ent.numel(), device=ln.device) - (upto[ent] - upto[e0])
        rows = torch.repeat_interleave(torch.arange(r0, r1, device=ln.device), rpA[r0 + 1:r1 + 1] - rpA[r0:r1])
        keys, order = torch.sort(rows[ent - e0] * n + ciB[at].long(), stable=True)
        yield r0, r1, keys, (vA[ent] * vB[at])[order]
        r0 = r1


def _multiply(A, B):
    """C = A*B as (rowptr, colidx, val) by sorting every product; 64 bits."""
    m, n = A[0], B[1]
    counts, cols, vals = [], [], []
    for r0, r1, keys, prods in _expand(A, B):
        uniq, where = torch.unique_consecutive(keys, return_inverse=True)
        rows = torch.div(uniq, n, rounding_mode="floor")
        counts.append(torch.bincount(rows - r0, minlength=r1 - r0))
        cols.append((uniq - rows * n).to(torch.int32))
        vals.append(torch.zeros(uniq.numel(), dtype=torch.float64, device=keys.device).index_add_(0, where, prods))
    rp = torch.zeros(m + 1, dtype=torch.int64, device=cols[0].device)
    rp[1:] = torch.cumsum(torch.cat(counts), 0)
    return rp.to(torch.int32), torch.cat(cols), torch.cat(vals)


def _sizes(pairs):
    """(4-byte words of the distinct operands as CSR, scalar products, entries
    of C) over the pairs."""
    words, prods, nnz = 0, 0, 0
    for A, B in pairs:
        for M in (A,) if B is A else (A, B):
            words += 3 * M[3].numel() + M[0] + 1
        for _, _, keys, _ in _expand(A, B):
            prods += keys.numel()
            nnz += int((keys[1:] != keys[:-1]).sum()) + (1 if keys.numel() else 0)
    return words, prods, nnz


def work(case):
    pairs = _operands(case, 1)
    if case["path"] == "order":
        A = pairs[0][0]
        words = 3 * A[3].numel() + A[0] + 1
        return {"bytes": 4 * (2 * words + A[0]), "flops": 0}  # the matrix in and out, and its order
    words, prods, nnz = _sizes(pairs)
    out = 3 * nnz + sum(A[0] + 1 for A, _ in pairs)
    return {"bytes": 4 * (words + out), "flops": 2 * prods}


def tolerance(case):
    """Orders and permuted copies are whole; a product's pattern too, its
    values sums of FP64 products: sums in another order (`exact` adds them in
    no order of its own) are up to 4.7e-16 off on the R-MAT graphs, the longest
    sums with the most cancellation; four times that."""
    if case["path"] == "order":
        return "exact"
    return {"rel": 2e-15, "max": 8e-14}


def exact(case, seed):
    if case["path"] == "order":
        return None  # an order has no value that another program would give
    got = [_multiply(A, B) for A, B in _operands(case, seed)]
    if case["path"] == "batch":
        return got
    if case["path"] == "host":
        return tuple(x.cpu().numpy() for x in got[0])
    return got[0]
