"""GPU orderings and bipermutations against the oracle (and, for original /
degree / RCM, against the reference's own order_utils.py outputs in
tests/golden/orders.npz); reorder plans; the reordered product restored."""
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
GOLD = Path(__file__).resolve().parent / "golden"


def _dev(mat):
    import torch
    m, n, rp, ci, v = mat
    d = torch.device("cuda", 0)
    return (torch.from_numpy(np.ascontiguousarray(rp, np.int32)).to(d),
            torch.from_numpy(np.ascontiguousarray(ci, np.int32)).to(d),
            torch.from_numpy(np.ascontiguousarray(v, np.float64)).to(d))


def _mats(gen):
    return {
        "lap": gen.laplacian_2d(40, 33),
        "st27": gen.stencil_27pt_3d(12, seed=2),
        "st27_perm": gen.permute_symmetric(gen.stencil_27pt_3d(10, seed=1), gen.random_symmetric_permutation(1000, 7)),
        "pois": gen.random_poisson(700, None, 5.0, seed=4),
        "rmat": gen.rmat(11, 8, seed=9),          # self loops, isolated vertices, hubs
        "rect": gen.random_poisson(300, 500, 4.0, seed=1),
    }


@pytest.mark.parametrize("kind", ["original", "degree", "random", "gray", "rcm"])
def test_gpu_orderings_match_oracle(tsg, ctx, oracle, gen, kind):
    for name, mat in _mats(gen).items():
        if kind == "rcm" and mat[0] != mat[1]:
            continue
        rp, ci, _ = _dev(mat)
        got = tsg.order(ctx, kind, mat[0], mat[1], rp, ci, seed=5).cpu().numpy()
        want = oracle.order(kind, mat, seed=5)
        np.testing.assert_array_equal(got, want, err_msg=f"{kind} on {name}")
        assert np.array_equal(np.sort(got), np.arange(mat[0]))


def test_orderings_match_reference_order_utils(tsg, ctx):
    z = np.load(GOLD / "orders.npz")
    for nm in sorted({k.split("/")[0] for k in z.files}):
        m, n = (int(x) for x in z[f"{nm}/m"])
        mat = (m, n, z[f"{nm}/rowptr"], z[f"{nm}/colidx"], z[f"{nm}/val"])
        rp, ci, _ = _dev(mat)
        for seed in (1, 7):
            got = tsg.order(ctx, "random", m, n, rp, ci, seed=seed).cpu().numpy()
            np.testing.assert_array_equal(got, z[f"{nm}/random{seed}"], err_msg=f"random/{seed} on {nm}")
        for kind in ("original", "degree", "rcm"):
            got = tsg.order(ctx, kind, m, n, rp, ci).cpu().numpy()
            if kind == "rcm" and nm == "rmat7":
                continue  # scipy seeds ties through an unstable argsort; see test_oracle_orders
            np.testing.assert_array_equal(got, z[f"{nm}/{kind}"], err_msg=f"{kind} on {nm}")


def test_permute_csr_matches_oracle(tsg, ctx, oracle, gen):
    import torch
    for name, mat in _mats(gen).items():
        m, n = mat[0], mat[1]
        rng = np.random.default_rng(3)
        row_old = rng.permutation(m).astype(np.int32)
        col_old = rng.permutation(n).astype(np.int32)
        col_new = np.empty(n, np.int32)
        col_new[col_old] = np.arange(n, dtype=np.int32)
        rp, ci, v = _dev(mat)
        d = torch.device("cuda", 0)
        orp, oci, ov = tsg.permute_csr(ctx, m, n, rp, ci, v, torch.from_numpy(row_old).to(d),
                                       torch.from_numpy(col_new).to(d))
        W = oracle.apply_bipermutation(mat, row_old, col_new)
        np.testing.assert_array_equal(orp.cpu().numpy(), W[2])
        np.testing.assert_array_equal(oci.cpu().numpy(), W[3])
        np.testing.assert_array_equal(ov.cpu().numpy(), W[4])


def test_dropin_apply_restore_round_trip(tsg, gen):
    mat = gen.random_poisson(333, 444, 6.0, seed=2)
    rng = np.random.default_rng(8)
    r, c = rng.permutation(333), rng.permutation(444)
    P = tsg.apply_bipermutation_csr(mat, r, c)
    back = tsg.restore_bipermutation_csr(P, r, c)
    for a, b in zip(back[2:], mat[2:]):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("algo", ["original", "rcm", "degree", "gray", "random"])
def test_reorder_plan_estimates_and_restored_product(tsg, ctx, oracle, gen, algo, monkeypatch):
    """AA plan on a randomly permuted 3D stencil: the plan's tile-count
    estimates equal the reference's sampled estimators (restated in the oracle,
    which tests/test_plan_estimates.py pins to the reference's own code) for
    the plan's permutations, and the product computed in the new order and
    restored equals the product of the original matrix."""
    monkeypatch.setenv("TASA_ENABLE_UNSAFE_RANDOM", "1")
    base = gen.stencil_27pt_3d(10, seed=3)
    mat = gen.permute_symmetric(base, gen.random_symmetric_permutation(1000, 11))
    plan = tsg.build_reorder_plan("AA", algo, mat)
    p = plan["row_perm"]
    assert np.array_equal(plan["inner_perm"], p) and np.array_equal(plan["col_perm"], p)
    if algo == "original":
        assert np.array_equal(p, np.arange(1000)) and plan["guard_degraded_to_identity"] == 1
    else:
        np.testing.assert_array_equal(p, oracle.order(algo, mat, seed=1))
    want = oracle.reorder_estimates("AA", mat, mat, p, p, p)
    assert {f: plan[f] for f in want} == want
    # product in the new order on the GPU, restored to the original order
    Cp, _ = tsg.spgemm_csr_host(ctx, tsg.apply_bipermutation_csr(mat, p, p))
    C = tsg.restore_bipermutation_csr(Cp, p, p)
    G = oracle.gustavson(mat, mat)
    np.testing.assert_array_equal(C[2], G[2])
    np.testing.assert_array_equal(C[3], G[3])
    rel = np.abs(C[4] - G[4]) / np.maximum(np.abs(G[4]), 1e-300)
    assert rel.max() <= 1e-12   # the inner index order changes with the ordering


def test_unknown_ordering_reports_missing_dependency(tsg, gen, monkeypatch):
    with pytest.raises(tsg.TsgError) as e:
        tsg.build_reorder_plan("AA", "slashburn", gen.laplacian_2d(8))
    assert e.value.status == -20
    # the reference's random adapter runs only when asked to (order_gen exits
    # 42 without TASA_ENABLE_UNSAFE_RANDOM=1, reported as -20)
    monkeypatch.delenv("TASA_ENABLE_UNSAFE_RANDOM", raising=False)
    with pytest.raises(tsg.TsgError) as e:
        tsg.build_reorder_plan("AA", "random", gen.laplacian_2d(8))
    assert e.value.status == -20
    monkeypatch.setenv("TASA_ENABLE_UNSAFE_RANDOM", "1")
    monkeypatch.setenv("TASA_RANDOM_SEED", "7")
    plan = tsg.build_reorder_plan("AA", "random", gen.laplacian_2d(8))
    import random
    want = list(range(64))
    random.Random(7).shuffle(want)
    np.testing.assert_array_equal(plan["row_perm"], want)


@pytest.mark.parametrize("kind", ["AAT", "AB"])
@pytest.mark.parametrize("algo", ["original", "rcm", "degree", "random"])
def test_reorder_plan_ab_and_aat(tsg, ctx, oracle, gen, kind, algo, monkeypatch):
    """A*A^T and A*B plans (src/external_reorder.h:204-321): rows and the inner
    axis take A's order, columns B's (A's for A*A^T); the plan's tile-count
    estimates equal the reference's sampled estimators for those
    permutations, and the product computed in the new order and restored
    equals the product of the original operands."""
    monkeypatch.setenv("TASA_ENABLE_UNSAFE_RANDOM", "1")
    n = 700
    base = gen.random_poisson(n, None, 5.0, seed=21)   # square, not symmetric
    A = gen.permute_symmetric(base, gen.random_symmetric_permutation(n, 4))
    B = gen.transpose(A) if kind == "AAT" else gen.permute_symmetric(gen.banded(n, 6, seed=2),
                                                                        gen.random_symmetric_permutation(n, 9))
    plan = tsg.build_reorder_plan(kind, algo, A, B)
    rp, ip, cp = plan["row_perm"], plan["inner_perm"], plan["col_perm"]
    np.testing.assert_array_equal(ip, rp)
    if algo == "original":
        assert np.array_equal(rp, np.arange(n)) and np.array_equal(cp, np.arange(n))
    else:
        np.testing.assert_array_equal(rp, oracle.order(algo, A, seed=1))
        np.testing.assert_array_equal(cp, rp if kind == "AAT" else oracle.order(algo, B, seed=1))
    assert plan["shared_symmetric_csr"] == 0
    want = oracle.reorder_estimates(kind, A, B, rp, ip, cp)
    assert {f: plan[f] for f in want} == want
    Cp, _ = tsg.spgemm_csr_host(ctx, tsg.apply_bipermutation_csr(A, rp, ip), tsg.apply_bipermutation_csr(B, ip, cp))
    C = tsg.restore_bipermutation_csr(Cp, rp, cp)
    G = oracle.gustavson(A, B)
    np.testing.assert_array_equal(C[2], G[2])
    np.testing.assert_array_equal(C[3], G[3])
    rel = np.abs(C[4] - G[4]) / np.maximum(np.abs(G[4]), 1e-300)
    assert rel.max(initial=0.0) <= 1e-12   # the inner index order changes with the ordering


@pytest.mark.parametrize("leaves", [2047, 2048, 2049, 6000])
def test_rcm_levels_with_large_buckets(tsg, ctx, oracle, leaves):
    """RCM of a hub whose level has one bucket below, at and above the size
    that the level kernel ranks by itself, with a path of narrow levels
    behind it, equals the oracle's."""
    import torch
    n = leaves + 40
    edges = [(0, i) for i in range(1, leaves + 1)] + [(leaves + i, leaves + i + 1) for i in range(39)]
    r = np.array([e for a, b in edges for e in (a, b)])
    c = np.array([e for a, b in edges for e in (b, a)])
    key = np.sort(r.astype(np.int64) * n + c)
    rp = np.searchsorted(key // n, np.arange(n + 1)).astype(np.int32)
    ci = (key % n).astype(np.int32)
    d = torch.device("cuda", torch.cuda.current_device())
    got = tsg.order(ctx, "rcm", n, n, torch.from_numpy(rp).to(d), torch.from_numpy(ci).to(d)).cpu().numpy()
    mat = (n, n, rp, ci, np.ones(ci.size))
    assert np.array_equal(got, oracle.order("rcm", mat))


@pytest.mark.parametrize("longest", [1, 33, 255, 256, 257, 900])
def test_permute_rows_up_to_and_past_the_ranked_length(tsg, ctx, longest):
    """Rows ranked in place (up to 256 entries) and whole-matrix sorts, repeated
    columns among them, against a stable numpy sort (copies: tolerance 0)."""
    import torch
    rng = np.random.default_rng(longest)
    m, n = 70, 1200
    counts = rng.integers(0, longest + 1, m)
    counts[11] = longest
    rp = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    ci = np.concatenate([np.sort(rng.choice(n, c, replace=bool(i % 3 == 0))) for i, c in enumerate(counts)]).astype(np.int32)
    v = rng.uniform(-1, 1, ci.size)
    row_old, col_new = rng.permutation(m).astype(np.int32), rng.permutation(n).astype(np.int32)
    d = torch.device("cuda", torch.cuda.current_device())
    got = tsg.permute_csr(ctx, m, n, *[torch.from_numpy(x).to(d) for x in (rp, ci, v, row_old, col_new)])
    rows = [np.arange(rp[o], rp[o + 1]) for o in row_old]
    at = np.concatenate([e[np.argsort(col_new[ci[e]], kind="stable")] for e in rows])
    np.testing.assert_array_equal(got[0].cpu().numpy(), np.concatenate([[0], np.cumsum(counts[row_old])]))
    np.testing.assert_array_equal(got[1].cpu().numpy(), col_new[ci[at]])
    np.testing.assert_array_equal(got[2].cpu().numpy(), v[at])


def test_rcm_of_patterns_that_are_not_symmetric_or_not_in_order(tsg, ctx, oracle, gen):
    """One entry without its mirror, a repeated one, rows out of order: the
    pattern is symmetrised by a sort, as before."""
    import torch
    d = torch.device("cuda", torch.cuda.current_device())
    m, n, rp, ci, v = gen.laplacian_2d(20)
    want = oracle.order("rcm", (m, n, rp, ci, v))

    def rcm(rp, ci):
        return tsg.order(ctx, "rcm", m, n, torch.from_numpy(rp).to(d), torch.from_numpy(ci).to(d)).cpu().numpy()

    assert np.array_equal(rcm(rp, ci), want)
    at = int(np.flatnonzero(ci[rp[50]:rp[51]] > 50)[0] + rp[50])  # drop (50, j): (j, 50) stays
    rp1 = rp.copy()
    rp1[51:] -= 1
    assert np.array_equal(rcm(rp1, np.delete(ci, at)), want)
    rp2 = rp.copy()
    rp2[51:] += 1
    assert np.array_equal(rcm(rp2, np.insert(ci, at, ci[at])), want)
    ci3 = ci.copy()
    ci3[rp[50]:rp[51]] = ci3[rp[50]:rp[51]][::-1]
    assert np.array_equal(rcm(rp, ci3), want)


@pytest.mark.parametrize("hubs,leaves", [(1, 1023), (1, 1024), (7, 1500), (40, 1100), (2, 60000)])
def test_rcm_of_vertices_with_many_neighbours(tsg, ctx, oracle, hubs, leaves):
    """Hubs around the number of neighbours that one warp expands, several in a
    level and one of most vertices, each joined to the first; leaves of two hubs
    among them; rows that a block checks and copies as a whole."""
    import torch
    rng = np.random.default_rng(hubs)
    n = 1 + hubs * (leaves + 1)
    first = 1 + np.arange(hubs) * (leaves + 1)
    edges = [np.stack([np.zeros(hubs, np.int64), first])]
    edges += [np.stack([np.full(leaves, h), h + 1 + np.arange(leaves)]) for h in first]
    if hubs > 1:
        edges.append(np.stack([rng.choice(first, 300), rng.integers(1, n, 300)]))
    a, b = np.concatenate(edges, axis=1)
    a, b = a[a != b], b[a != b]
    diag = rng.choice(n, n // 3, replace=False)  # some diagonal entries
    key = np.unique(np.concatenate([a * n + b, b * n + a, diag * n + diag]))
    rp = np.searchsorted(key // n, np.arange(n + 1)).astype(np.int32)
    ci = (key % n).astype(np.int32)
    d = torch.device("cuda", torch.cuda.current_device())
    used = ctx.pool_used()
    got = tsg.order(ctx, "rcm", n, n, torch.from_numpy(rp).to(d), torch.from_numpy(ci).to(d)).cpu().numpy()
    assert np.array_equal(got, oracle.order("rcm", (n, n, rp, ci, np.ones(ci.size))))
    ctx.synchronize()
    assert ctx.pool_used() <= used


@pytest.mark.parametrize("longest", [30, 900])
def test_permute_csr_in_a_captured_graph(tsg, oracle, gen, longest):
    """The C call may be captured: the graph's replay permutes what its inputs
    hold then."""
    import ctypes
    import torch
    rng = np.random.default_rng(longest)
    m, n = 300, 1000
    counts = rng.integers(0, 31, m)
    counts[5] = longest
    rp = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    ci = np.concatenate([np.sort(rng.choice(n, c, replace=False)) for c in counts]).astype(np.int32)
    d = torch.device("cuda", 0)
    row_old, col_new = rng.permutation(m).astype(np.int32), rng.permutation(n).astype(np.int32)
    dev = [torch.from_numpy(x).to(d) for x in (rp, ci, np.zeros(ci.size), row_old, col_new)]
    out = [torch.empty(m + 1, dtype=torch.int32, device=d), torch.empty(ci.size, dtype=torch.int32, device=d),
           torch.empty(ci.size, dtype=torch.float64, device=d)]
    stream = torch.cuda.Stream()
    ctx = tsg.Context(0, stream=stream.cuda_stream)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        tsg.check(tsg.lib().tsg_permute_csr(ctx.handle, m, n, ci.size, *[ctypes.c_void_p(t.data_ptr()) for t in dev + out]))
    for seed in (1, 2):
        v = np.random.default_rng(seed).uniform(-1, 1, ci.size)
        dev[2].copy_(torch.from_numpy(v))
        graph.replay()
        torch.cuda.synchronize()
        want = oracle.apply_bipermutation((m, n, rp, ci, v), row_old, col_new)
        for got, w in zip(out, want[2:]):
            np.testing.assert_array_equal(got.cpu().numpy(), w)
    del graph
    ctx.close()
