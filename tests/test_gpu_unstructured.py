"""Products whose rows are uneven or wide -- step 1 by a CTA per tile row with
its bitmaps kept, step 2 of wide rows in parts, step 3 by column windows --
and the dense tile kernel, against the oracle at the sizes where each changes:
window and table-block edges, heavy rows around WIN_HEAVY (256) entries, tile
rows around one part (1,024 entries), columns past one pass of step 2 (98,304)
and past what step 1 keeps (262,144) or holds at once (1,048,576), an A with
no row view.  Values bit for bit: the order of the sums is the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rows(m, n, counts, seed, hub=0):
    """Rows of counts[i] distinct random columns; hub: every row holds column 0 too."""
    rng = np.random.default_rng(seed)
    cols = []
    for c in counts:
        x = np.unique(rng.integers(0, n, int(c) * 2))
        x = np.sort(rng.choice(x, min(int(c), x.size), replace=False)) if c else x[:0]
        if hub and c:
            x = np.unique(np.concatenate([[0], x]))
        cols.append(x)
    rp = np.concatenate([[0], np.cumsum([x.size for x in cols])]).astype(np.int32)
    ci = np.concatenate(cols).astype(np.int32)
    return m, n, rp, ci, rng.uniform(-1, 1, ci.size)


def _tiled(tsg, ctx, mat, flags):
    import torch
    d = torch.device("cuda", torch.cuda.current_device())
    m, n, rp, ci, v = mat
    return tsg.csr_to_tiled(ctx, m, n, *[torch.from_numpy(x).to(d) for x in (rp, ci, v)], flags)


def _same(got, want):
    assert np.array_equal(got[0], want[2])
    assert np.array_equal(got[1], want[3])
    both_nan = np.isnan(got[2]) & np.isnan(want[4])
    assert np.array_equal(got[2].view(np.uint64)[~both_nan], want[4].view(np.uint64)[~both_nan])


def _check(tsg, ctx, oracle, A, B, flagsA):
    tA, tB = _tiled(tsg, ctx, A, flagsA), _tiled(tsg, ctx, B, tsg.TSG_TILED_CSC_VIEW)
    C, info = tsg.spgemm(ctx, tA, tB)
    _same([x.cpu().numpy() for x in tsg.tiled_to_csr(ctx, C)], oracle.gustavson(A, B, nthreads=8))
    if C.numtile < 400000:
        got = C.download()
        want = oracle.spgemm_tiled(oracle.csr2tile_row_major(A), oracle.csr2tile_col_major(B))
        for k in ("tile_ptr", "tile_columnidx", "tile_rowidx", "tile_nnz", "tile_csr_Ptr", "tile_csr_Col", "mask"):
            np.testing.assert_array_equal(got[k], want[k], err_msg=k)
    for t in (tA, tB, C):
        t.free()
    return info


def _case(name):
    rng = np.random.default_rng(7)
    if name.startswith("cols"):  # window and block edges
        n = int(name[4:])
        return _rows(70, 300, rng.integers(0, 60, 70), 1), _rows(300, n, rng.integers(0, min(n // 2, 26) + 1, 300), 2, hub=1)
    if name == "heavy":  # rows around WIN_HEAVY entries among light ones, every B row holding column 0
        counts = [255, 0, 257, 3, 256, 40, 700, 1, 2, 5, 0, 258, 9, 9, 9, 9, 600, 4]
        return _rows(18, 1500, counts, 3), _rows(1500, 1300, rng.integers(0, 30, 1500), 4, hub=1)
    if name == "heavy among light":  # ... where the mean row is short
        counts = [255, 0, 257, 3, 256, 40, 700, 1, 2, 5, 0, 258, 9, 9, 9, 9, 600, 4] + [2] * 300
        return _rows(318, 1500, counts, 3), _rows(1500, 1300, rng.integers(0, 30, 1500), 4, hub=1)
    if name == "parts":  # tile rows of 1, 2 and 5 parts
        counts = [63] * 16 + [64] * 16 + [65] * 16 + [257] * 16 + [3] * 5
        return _rows(69, 4000, counts, 5), _rows(4000, 5000, rng.integers(0, 12, 4000), 6)
    if name == "coarse table":  # 70,000 x 300,000: a table block wider than a heavy row's part; step 2 in passes
        long = [40 * i for i in range(400)]
        counts = np.zeros(70000, int)
        counts[long] = 2500  # rows of B that all of A meets
        rows = [np.sort(rng.choice(long, k, replace=False)) for k in [30] * 39 + [390]]
        rp = np.concatenate([[0], np.cumsum([r.size for r in rows])]).astype(np.int32)
        A = 40, 70000, rp, np.concatenate(rows).astype(np.int32), rng.uniform(-1, 1, rp[-1])
        return A, _rows(70000, 300000, counts, 9)
    assert name == "step 1 in passes"
    return _rows(33, 400, rng.integers(1, 40, 33), 10), _rows(400, 1100000, np.full(400, 300), 11)


@pytest.mark.parametrize("name", ["cols15", "cols255", "cols256", "cols257", "cols1024", "cols1025", "cols2000", "heavy",
                                  "heavy among light", "parts", "coarse table", "step 1 in passes"])
@pytest.mark.parametrize("view", [True, False])
def test_uneven_products(tsg, ctx, oracle, name, view):
    A, B = _case(name)
    flags = tsg.TSG_TILED_CSC_VIEW if view else tsg.TSG_TILED_PACKED_COL
    ctx.set_schedule("spa", dense=257)  # never the tile kernel
    try:
        info = _check(tsg, ctx, oracle, A, B, flags)
    finally:
        ctx.set_schedule("spa", dense=0)
    assert (info["step3_name"] == "k_step3_win") == (name != "step 1 in passes")


def test_window_step_on_tile_row_ranges(tsg, ctx, oracle, gen):
    """The host call computes a skewed product in ranges of tile rows."""
    mat = gen.rmat(12, 24, seed=5)
    out = tsg.HostResultBuffers(mat[0], 1 << 24)
    got, info = tsg.spgemm_csr_host_overlap(ctx, mat, None, out)
    assert info["nnz_C"] > 2 << 20  # more than one chunk
    assert info["step3_name"] == "k_step3_win"
    _same(got[2:], oracle.gustavson(mat, mat, nthreads=8))


def test_batch_of_uneven_products(tsg, ctx, oracle, gen):
    """Windows with heavy rows, hypersparse rows, dense tiles and an empty product
    in one batch (the SPA kernel's rows in a batch: test_hypersparse_rows_among_others)."""
    empty = (20, 300, np.zeros(21, np.int32), np.zeros(0, np.int32), np.zeros(0))
    mats = [_case("heavy"), _case("cols257"), _case("parts"), (gen.rmat(11, 12, seed=2), gen.rmat(11, 12, seed=3)),
            (gen.random_poisson(8192, 8192, 4.0, seed=10), gen.random_poisson(8192, 8192, 4.0, seed=11)),
            (gen.banded(400, 40, seed=1), gen.banded(400, 30, seed=2)), (empty, _case("cols257")[1])]
    pairs = [tuple(_tiled(tsg, ctx, x, tsg.TSG_TILED_CSC_VIEW) for x in ab) for ab in mats]
    batch = tsg.Batch(ctx, pairs)
    for _ in range(2):
        batch.run()
        batch.sync()
        for p, (a, b) in enumerate(mats):
            _same([x.cpu().numpy() for x in tsg.tiled_to_csr(ctx, batch.product(p))], oracle.gustavson(a, b, nthreads=8))
    batch.close()


@pytest.mark.parametrize("half", [7, 8, 20, 41])
@pytest.mark.parametrize("special", [None, np.inf, -np.inf, np.nan])
def test_dense_tiles_with_values_that_zero_does_not_absorb(tsg, ctx, oracle, gen, half, special):
    """Bands on both sides of the dense tile path (64 values of an A tile),
    ragged last tiles, and infinite or NaN values, whose product with an
    absent entry must not be formed."""
    A, B = gen.banded(203, half, seed=1), gen.banded(203, 30, seed=2)
    if special is not None:
        A[4][[5, 700, -3]] = special
        B[4][[9, 2000]] = special
    ctx.set_schedule("spa", dense=1)  # every product takes the tile kernel
    try:
        _check(tsg, ctx, oracle, A, B, tsg.TSG_TILED_CSC_VIEW)
    finally:
        ctx.set_schedule("spa", dense=0)


@pytest.mark.parametrize("n,entries", [(520, 520), (600, 600), (530, 40), (530, 8)])
def test_rows_of_many_tile_pairs(tsg, ctx, oracle, n, entries):
    """33 and 38 tiles a row on both sides (1,089 and 1,444 pairs, at most 128 C
    tiles): full rows, whose masks a warp makes pair by pair, and sparse ones,
    left to the CTA of wide rows."""
    A, B = _rows(n, n, [entries] * n, 1), _rows(n, n, [entries] * n, 2)
    for fused in (True, False):
        ctx.set_fusion(fused)
        try:
            _check(tsg, ctx, oracle, A, B, tsg.TSG_TILED_CSC_VIEW)
        finally:
            ctx.set_fusion(True)
    pairs = [tuple(_tiled(tsg, ctx, x, tsg.TSG_TILED_CSC_VIEW) for x in (A, B))]
    for sched in ("spa", "tiles", "elems"):
        batch = tsg.Batch(ctx, pairs, sched)
        batch.run()
        batch.sync()
        _same([x.cpu().numpy() for x in tsg.tiled_to_csr(ctx, batch.product(0))], oracle.gustavson(A, B, nthreads=8))
        batch.close()


@pytest.mark.parametrize("entries", [1, 4, 5, 6, 12])
def test_spa_rows_whose_products_meet(tsg, ctx, oracle, entries):
    """B rows of a few entries in 60 columns far apart, so that a batch of
    products meets most columns several times: batches of few entries (added
    entry by entry) and of many."""
    rng = np.random.default_rng(entries)
    hubs = np.sort(rng.choice(2500, 60, replace=False)) * 16 + 5
    A = _rows(70, 500, [40] * 70, 1)
    rows = [np.sort(rng.choice(hubs, entries if i % 7 else 1, replace=False)) for i in range(500)]
    rp = np.concatenate([[0], np.cumsum([r.size for r in rows])]).astype(np.int32)
    B = 500, 40000, rp, np.concatenate(rows).astype(np.int32), rng.uniform(-1, 1, rp[-1])
    assert _check(tsg, ctx, oracle, A, B, tsg.TSG_TILED_CSC_VIEW)["step3_name"] == "k_step3_spa<flat>"


def _mixed(tile_rows, seed, every=6):
    """Wide C tile rows, one in `every` with several values a tile and the others
    hypersparse, too few values a window for the window step."""
    m = 16 * tile_rows - 11
    A = _rows(m, 4000, [300 if i // 16 % every == 1 else 3 for i in range(m)], seed)
    return A, _rows(4000, 64000, [4] * 4000, seed + 1)


@pytest.mark.parametrize("dense", [257, 0])
def test_hypersparse_rows_among_others(tsg, ctx, oracle, dense):
    A, B = _mixed(14, 1)
    ctx.set_schedule("spa", dense=dense)
    try:
        info = _check(tsg, ctx, oracle, A, B, tsg.TSG_TILED_CSC_VIEW)
    finally:
        ctx.set_schedule("spa", dense=0)
    assert info["step3_name"] == "k_step3_spa<flat>"
    batch = tsg.Batch(ctx, [tuple(_tiled(tsg, ctx, x, tsg.TSG_TILED_CSC_VIEW) for x in (A, B))] * 2)
    for _ in range(2):
        batch.run()
        batch.sync()
        for p in range(2):
            _same([x.cpu().numpy() for x in tsg.tiled_to_csr(ctx, batch.product(p))], oracle.gustavson(A, B, nthreads=8))
    batch.close()


def test_hypersparse_rows_among_others_on_tile_row_ranges(tsg, ctx, oracle):
    A, B = _mixed(1100, 3, every=9)
    out = tsg.HostResultBuffers(A[0], 1 << 22)
    got, info = tsg.spgemm_csr_host_overlap(ctx, A, B, out)
    assert info["nnz_C"] > 2 << 20 and info["step3_name"] == "k_step3_spa<flat>"
    # a kernel of its own takes the hypersparse rows: enough tiles, few values in them
    assert info["numtile_C"] >= 1 << 17 and info["nnz_C"] < 4 * info["numtile_C"]
    _same(got[2:], oracle.gustavson(A, B, nthreads=8))


@pytest.mark.parametrize("m,e,wins", [(300, 60, False), (2000, 60, True)])
def test_few_rows_of_a_do_not_pay_for_tables_of_a_large_b(tsg, ctx, oracle, m, e, wins):
    """The windows' tables cost every row of B: 130 words of them a value of C
    are too many, 20 are not."""
    A, B = _rows(m, 100000, [e] * m, 1), _rows(100000, 40000, [12] * 100000, 2)
    ctx.synchronize()
    used = ctx.pool_used()
    info = _check(tsg, ctx, oracle, A, B, tsg.TSG_TILED_CSC_VIEW)
    assert (info["step3_name"] == "k_step3_win") == wins
    ctx.synchronize()
    assert ctx.pool_used() <= used


@pytest.mark.parametrize("entries,n", [(1, 98304), (1, 98320), (1, 300000), (3, 300000), (40, 300000), (200, 300000)])
def test_few_tiles_over_many_columns(tsg, ctx, oracle, entries, n):
    """Wide rows of few C tiles on both sides of what a pass of step 2 holds by
    columns (98,304), by a slot per tile, and of too many for that."""
    A, B = _rows(70, 2000, [entries] * 69 + [60], 1), _rows(2000, n, [1 + entries % 7] * 2000, 2)
    _check(tsg, ctx, oracle, A, B, tsg.TSG_TILED_CSC_VIEW)
    batch = tsg.Batch(ctx, [tuple(_tiled(tsg, ctx, x, tsg.TSG_TILED_CSC_VIEW) for x in (A, B))])
    batch.run()
    batch.sync()
    _same([x.cpu().numpy() for x in tsg.tiled_to_csr(ctx, batch.product(0))], oracle.gustavson(A, B, nthreads=8))
    batch.close()


def test_products_that_fail_leave_no_scratch(tsg, ctx):
    """C past 32-bit offsets is refused after steps 1 and 2, whose scratch goes."""
    n = 50000
    A = n, 16, np.arange(n + 1, dtype=np.int32), np.zeros(n, np.int32), np.ones(n)
    B = 16, n, np.array([0] + [n] * 16, np.int32), np.arange(n, dtype=np.int32), np.ones(n)
    tA, tB = _tiled(tsg, ctx, A, tsg.TSG_TILED_CSC_VIEW), _tiled(tsg, ctx, B, tsg.TSG_TILED_CSC_VIEW)
    ctx.synchronize()
    used = ctx.pool_used()
    for _ in range(2):
        with pytest.raises(tsg.TsgError) as e:
            tsg.spgemm(ctx, tA, tB)
        assert e.value.status == tsg.TSG_ERR_OVERFLOW
        del e
    import gc
    gc.collect()
    ctx.synchronize()
    assert ctx.pool_used() <= used
    for t in (tA, tB):
        t.free()


@pytest.mark.parametrize("n,wins", [(20000, False), (2000, True)])
def test_windows_that_c_does_not_fill(tsg, ctx, oracle, gen, n, wins):
    """A band times random rows: each C tile row meets about 230 tile columns,
    12 of a window's 64 over 20,000 columns and all of them over 2,000."""
    A, B = gen.banded(n, 16, seed=1), gen.random_poisson(n, n, 8.0, seed=2)
    info = _check(tsg, ctx, oracle, A, B, tsg.TSG_TILED_CSC_VIEW)
    assert (info["step3_name"] == "k_step3_win") == wins
