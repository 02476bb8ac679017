"""Learned choice of ordering and accumulator setting for the tiled SpGEMM.

A small FP32 MLP (features -> 64 -> 64 -> one output per configuration),
trained and evaluated by the library's own CUDA kernels (tsg_mlp_*),
predicts the relative log run time of every (ordering, accumulator)
configuration of C = A*A from cheap matrix features; the selector runs the
argmin.  Training data is generated by the method itself: every candidate
configuration is timed on the GPU over seeded synthetic matrices.  The
exhaustive search (time everything, keep the best) is both the fallback --
used whenever the model is absent or a matrix's features fall outside the
training range -- and the yardstick of the model's regret.
"""
from __future__ import annotations

import ctypes
import math
import time
from dataclasses import dataclass

import numpy as np

from . import (ORDER_KINDS, TSG_TILED_CSC_VIEW, Context, build_reorder_plan, check, csr_to_tiled, lib, order,
               permute_csr, product_bounds, reorder_estimates, spgemm)

# "tasa": the tile-aware planner (build_reorder_plan), whose general plans
# give the rows, inner axis and columns different orders
ORDERINGS = ["original", "rcm", "degree", "gray", "random", "tasa"]
ACCUMULATORS = [("spa", 8, 512), ("tiles", 8, 512), ("rows", 8, 256)]
CONFIGS = [(o, a) for o in ORDERINGS for a in ACCUMULATORS]
NFEAT = 25


def _declare(L):
    vp, ip = ctypes.c_void_p, ctypes.c_int
    L.tsg_row_features.argtypes = [vp, ip, vp, vp, ctypes.POINTER(ctypes.c_ulonglong)]
    L.tsg_mlp_create.argtypes = [vp, ip, ip, ip, ctypes.c_ulonglong, ctypes.POINTER(vp)]
    L.tsg_mlp_destroy.argtypes = [vp]
    L.tsg_mlp_num_params.argtypes = [vp]
    L.tsg_mlp_train_step.argtypes = [vp, ip, vp, vp, vp, ctypes.c_float, ctypes.POINTER(ctypes.c_float)]
    L.tsg_mlp_forward.argtypes = [vp, ip, vp, vp]
    L.tsg_mlp_get.argtypes = [vp, ip, vp]
    L.tsg_mlp_set.argtypes = [vp, vp]


_declared = False


def _lib():
    global _declared
    L = lib()
    if not _declared:
        _declare(L)
        _declared = True
    return L


# ---------------------------------------------------------------------------
# features
# ---------------------------------------------------------------------------
def _dev(mat, device):
    import torch
    m, n, rp, ci, v = mat
    d = torch.device("cuda", device)
    return (torch.from_numpy(np.ascontiguousarray(rp, np.int32)).to(d),
            torch.from_numpy(np.ascontiguousarray(ci, np.int32)).to(d),
            torch.from_numpy(np.ascontiguousarray(v, np.float64)).to(d))


def features(ctx: Context, mat, device=0, dev=None, tiled=None) -> np.ndarray:
    """Feature vector of C = A*A for matrix A (25 floats): row statistics,
    tile counts and bounds, and the reorder planner's sampled C-tile estimate
    (24 strided tile rows, src/reorder.h:890-929) per A tile and per tile row."""
    m, n = mat[0], mat[1]
    rp, ci, v = dev if dev is not None else _dev(mat, device)
    raw = (ctypes.c_ulonglong * 24)()
    check(_lib().tsg_row_features(ctx.handle, int(m), ctypes.c_void_p(rp.data_ptr()),
                                  ctypes.c_void_p(ci.data_ptr()), raw))
    raw = np.array(raw[:], dtype=np.float64)
    T = tiled if tiled is not None else csr_to_tiled(ctx, m, n, rp, ci, v, TSG_TILED_CSC_VIEW)
    prods, pairs = product_bounds(ctx, T, T)
    nnz = max(raw[0], 1.0)
    avg = raw[0] / max(m, 1)
    var = max(raw[1] / max(m, 1) - avg * avg, 0.0)
    hist = raw[6:18] / max(m, 1)
    tilem, tilen, nt = T.s.tilem, T.s.tilen, max(T.s.numtile, 1)
    f = [
        math.log2(max(n, 1)), math.log2(nnz + 1), math.log2(avg + 1), math.sqrt(var) / max(avg, 1e-9),
        math.log2(raw[2] + 1) - math.log2(avg + 1), raw[3] / nnz / max(n, 1), raw[4] / max(n, 1), raw[5] / max(m, 1),
        hist[0], hist[1], hist[2], hist[3], hist[4], hist[5], hist[6], hist[7] + hist[8] + hist[9] + hist[10] + hist[11],
        raw[18] / nnz, math.log2(nt / max(tilem * tilen, 1)), math.log2(nnz / nt), math.log2(max(prods, 1) / nnz),
        math.log2(max(pairs, 1) / nt), math.log2(nt + 1), math.log2(max(prods, 1)),
    ]
    ident = np.arange(m)
    est_c = reorder_estimates("AA", mat, None, ident, ident, ident)["estimated_c_tiles_before"] if m == n else nt
    f += [math.log2(max(est_c, 1) / nt), math.log2(max(est_c, 1) / max(tilem, 1))]
    if tiled is None:
        T.free()
    return np.array(f, dtype=np.float32)


# ---------------------------------------------------------------------------
# method-generated timings
# ---------------------------------------------------------------------------
def time_configs(ctx: Context, mat, device=0, repeats=3, seed=1):
    """Run time (ms, steps 1-3) of C = A*A for every configuration, and the
    ordering cost (ms) of every ordering (plan and permutation of the CSR;
    "tasa" multiplies P_r A P_i^T by P_i A P_c^T when its axes differ)."""
    import torch
    m, n = mat[0], mat[1]
    rp, ci, v = _dev(mat, device)
    ctx.set_timing(True)
    times = np.zeros(len(CONFIGS))
    order_ms = {}
    feats = None
    for oi, oname in enumerate(ORDERINGS):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        if oname == "tasa":
            plan = build_reorder_plan("AA", "tasa", mat, symmetric=_pattern_symmetric(mat))
            axes = [torch.from_numpy(np.ascontiguousarray(plan[a], np.int32)).to(rp.device)
                    for a in ("row_perm", "inner_perm", "col_perm")]
        else:
            axes = [order(ctx, oname, m, n, rp, ci, seed=seed)] * 3
        news = []
        for perm in axes:
            new = torch.empty_like(perm)
            new[perm.long()] = torch.arange(m, dtype=torch.int32, device=perm.device)
            news.append(new)
        same = all(torch.equal(axes[0], a) for a in axes[1:])
        pa = permute_csr(ctx, m, n, rp, ci, v, axes[0], news[1])
        pb = pa if same else permute_csr(ctx, m, n, rp, ci, v, axes[1], news[2])
        torch.cuda.synchronize()
        order_ms[oname] = (time.perf_counter() - t0) * 1e3
        T = csr_to_tiled(ctx, m, n, *pa, TSG_TILED_CSC_VIEW)
        TB = T if same else csr_to_tiled(ctx, m, n, *pb, TSG_TILED_CSC_VIEW)
        if oname == "original":
            feats = features(ctx, mat, device, dev=(rp, ci, v), tiled=T)
        for ai, acc in enumerate(ACCUMULATORS):
            ctx.set_schedule(*acc)
            best = float("inf")
            for _ in range(repeats):
                C, info = spgemm(ctx, T, TB)
                best = min(best, info["ms_total"])
                C.free()
            times[oi * len(ACCUMULATORS) + ai] = best
        if TB is not T:
            TB.free()
        T.free()
    ctx.set_schedule(*ACCUMULATORS[0])
    ctx.set_timing(False)
    return feats, times, order_ms


def _pattern_symmetric(mat) -> bool:
    """Whether the pattern equals its transpose (what a symmetric Matrix
    Market file declares)."""
    m, n, rp, ci, _ = mat
    if m != n:
        return False
    rows = np.repeat(np.arange(m, dtype=np.int64), np.diff(np.asarray(rp, np.int64)))
    cols = np.asarray(ci, np.int64)
    a = np.sort(rows * n + cols)
    b = np.sort(cols * n + rows)
    return a.size == b.size and bool(np.array_equal(a, b))


def training_matrices(gen, count, seed=0):
    """Seeded synthetic matrices from several families, half of them under a
    random symmetric permutation (the case orderings are for)."""
    rng = np.random.default_rng(seed)
    out = []
    for i in range(count):
        fam = int(rng.integers(0, 5))
        s = int(rng.integers(0, 2**31 - 1))
        if fam == 0:
            mat = gen.laplacian_2d(int(rng.integers(40, 220)))
        elif fam == 1:
            mat = gen.stencil_27pt_3d(int(rng.integers(10, 30)), seed=s)
        elif fam == 2:
            mat = gen.banded(int(rng.integers(2000, 40000)), int(rng.integers(3, 40)), seed=s)
        elif fam == 3:
            mat = gen.random_poisson(int(rng.integers(2000, 40000)), None, float(rng.uniform(2, 14)), seed=s)
        else:
            mat = gen.rmat(int(rng.integers(10, 14)), int(rng.integers(4, 16)), seed=s)
        if fam in (0, 1, 2) and rng.random() < 0.6:
            mat = gen.permute_symmetric(mat, gen.random_symmetric_permutation(mat[0], s % 100000))
        out.append(mat)
    return out


# ---------------------------------------------------------------------------
# the network
# ---------------------------------------------------------------------------
FIT_SPAN = np.e


class MLP:
    """tsg_mlp wrapper: FP32 F -> H -> H -> O network on the GPU."""

    def __init__(self, ctx: Context, F=NFEAT, H=64, O=len(CONFIGS), seed=1):
        self.ctx, self.F, self.H, self.O = ctx, F, H, O
        self.h = ctypes.c_void_p()
        check(_lib().tsg_mlp_create(ctx.handle, F, H, O, ctypes.c_ulonglong(seed), ctypes.byref(self.h)))
        self.nparam = _lib().tsg_mlp_num_params(self.h)
        self.mu = np.zeros(F, np.float32)
        self.sd = np.ones(F, np.float32)
        self.lo = None
        self.hi = None

    def params(self, which=0):
        out = np.zeros(self.nparam, np.float32)
        check(_lib().tsg_mlp_get(self.h, which, out.ctypes.data))
        return out

    def set_params(self, w):
        w = np.ascontiguousarray(w, np.float32)
        check(_lib().tsg_mlp_set(self.h, w.ctypes.data))

    def step(self, X, T, M=None, lr=1e-3):
        """One minibatch step on device tensors; returns the loss."""
        loss = ctypes.c_float(0)
        check(_lib().tsg_mlp_train_step(self.h, int(X.shape[0]), ctypes.c_void_p(X.data_ptr()),
                                        ctypes.c_void_p(T.data_ptr()),
                                        ctypes.c_void_p(M.data_ptr()) if M is not None else None, ctypes.c_float(lr),
                                        ctypes.byref(loss)))
        return loss.value

    def forward(self, X):
        import torch
        Y = torch.empty((X.shape[0], self.O), dtype=torch.float32, device=X.device)
        check(_lib().tsg_mlp_forward(self.h, int(X.shape[0]), ctypes.c_void_p(X.data_ptr()),
                                     ctypes.c_void_p(Y.data_ptr())))
        self.ctx.synchronize()
        return Y

    def fit(self, feats, targets, epochs=300, batch=64, lr=2e-3, seed=0, device=0):
        """Trains on relative log run times (each row minus its mean).  A time
        above FIT_SPAN times the row's best counts as that: how much slower the
        slow ones are is not asked, and fitting it costs the choice among the
        near ones (held-out regret of 64 matrices' timings, mean and worst of 12
        fits: 0.077 and 0.105 without, 0.058 and 0.069 with it)."""
        import torch
        self.mu = feats.mean(0).astype(np.float32)
        self.sd = (feats.std(0) + 1e-6).astype(np.float32)
        self.lo, self.hi = feats.min(0), feats.max(0)
        X = ((feats - self.mu) / self.sd).astype(np.float32)
        Y = np.log(np.minimum(targets, FIT_SPAN * targets.min(1, keepdims=True)))
        Y = (Y - Y.mean(1, keepdims=True)).astype(np.float32)
        d = torch.device("cuda", device)
        Xd, Yd = torch.from_numpy(X).to(d), torch.from_numpy(Y).to(d)
        rng = np.random.default_rng(seed)
        losses = []
        for ep in range(epochs):
            perm = rng.permutation(X.shape[0])
            tot = 0.0
            for s in range(0, X.shape[0], batch):
                idx = torch.from_numpy(perm[s:s + batch]).to(d)
                tot += self.step(Xd[idx].contiguous(), Yd[idx].contiguous(), lr=lr) * len(idx)
            losses.append(tot / X.shape[0])
        return losses

    def predict(self, feats):
        import torch
        X = ((np.atleast_2d(feats) - self.mu) / self.sd).astype(np.float32)
        return self.forward(torch.from_numpy(X).to(torch.device("cuda", torch.cuda.current_device()))).cpu().numpy()

    def in_range(self, f, slack=0.5):
        if self.lo is None:
            return False
        span = np.maximum(self.hi - self.lo, 1e-6)
        return bool(np.all(f >= self.lo - slack * span) and np.all(f <= self.hi + slack * span))

    def close(self):
        if self.h:
            _lib().tsg_mlp_destroy(self.h)
            self.h = ctypes.c_void_p()


@dataclass
class Choice:
    config: tuple
    source: str  # "model" or "exhaustive"


def choose(model: MLP | None, ctx: Context, mat, device=0) -> Choice:
    """The model's configuration, or the exhaustive search's when there is no
    model or the matrix lies outside the training range."""
    f = features(ctx, mat, device)
    if model is not None and model.in_range(f):
        return Choice(CONFIGS[int(np.argmin(model.predict(f)[0]))], "model")
    _, t, _ = time_configs(ctx, mat, device)
    return Choice(CONFIGS[int(np.argmin(t))], "exhaustive")


def regret(times, picks):
    """Mean and worst relative slowdown of picks (indices) vs the best."""
    best = times.min(1)
    got = times[np.arange(times.shape[0]), picks]
    r = got / best - 1.0
    return float(r.mean()), float(np.median(r)), float(r.max())
