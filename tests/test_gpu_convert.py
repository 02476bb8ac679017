"""Tiles -> CSR (k_t2c): a matrix that goes into tiles and out again is the
matrix it was, bit for bit (copies: tolerance 0), at the sizes where the
kernel's steps end: ragged last tile rows, full tiles (counts of 256), more
tiles in a tile row than one step or one 16-bit sum holds, tile rows that
choose each block size, and row offsets off their 16-byte boundary."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _matrix(kind, m, n, per_row, seed=3):
    rng = np.random.default_rng(seed)
    if kind == "full":
        counts = np.full(m, n)
    elif kind == "some":  # rows with nothing among them
        counts = np.where(rng.random(m) < 0.3, 0, rng.integers(0, min(n, per_row) + 1, m))
    else:
        counts = np.full(m, min(n, per_row))
        if kind == "hubs":  # rows of n / 20 entries in every 40th tile row and the last row
            counts[7::640] = counts[-1] = n // 20
    cols = [np.sort(rng.choice(n, c, replace=False)) if c < n else np.arange(n) for c in counts]
    rp = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    ci = np.concatenate(cols).astype(np.int32) if rp[-1] else np.zeros(0, np.int32)
    return m, n, rp, ci, rng.uniform(-1, 1, ci.size)


SHAPES = [
    ("full", 1, 1, 0), ("full", 17, 33, 0), ("full", 47, 16, 0), ("some", 31, 700, 40),
    ("some", 5000, 600, 9),            # few values a tile row: a half-warp each
    ("some", 16 * 2400 + 5, 300, 3),
    ("each", 600, 600, 4), ("each", 600, 600, 5),  # on both sides of 64 values a tile row
    ("each", 5000, 600, 9),            # narrow tile rows, 256 threads
    ("each", 16 * 2400 + 5, 600, 28),  # many of 448 values, a half-warp each ...
    ("each", 16 * 2400 + 5, 600, 29),  # ... and of 464, 128 threads
    ("hubs", 16 * 2400 + 5, 16 * 300, 2),  # long tile rows among them, the last too
    ("each", 33, 16 * 900, 400),       # wide, several steps of 512 tiles, most tiles empty in a row
    ("each", 16, 16 * 1100000, 80000), # one tile row of > 2048 steps: the 16-bit sums are emptied
    ("each", 48, 900, 31), ("each", 48, 900, 32), ("each", 37, 16 * 1024 + 5, 33),  # around 512 entries a tile row
    ("full", 37, 700, 0),              # a CTA each, full tiles, ragged
    ("each", 69, 16 * 4000, 2), ("each", 69, 16 * 4000, 3),  # on both sides of 32 tiles a tile row
    ("each", 27, 16 * 300000, 74), ("each", 27, 16 * 300000, 78),  # and of 4 entries for every 1,024 tile columns
    ("hubs", 33, 16 * 70000, 1),       # rows of very different length, passes with gaps between them
]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "-".join(map(str, s)))
@pytest.mark.parametrize("off_boundary", [False, True])
def test_tiles_and_back(tsg, ctx, oracle, shape, off_boundary):
    import torch
    m, n, rp, ci, v = _matrix(*shape)
    d = torch.device("cuda", torch.cuda.current_device())
    dev = [torch.from_numpy(x).to(d) for x in (rp, ci, v)]
    T = tsg.csr_to_tiled(ctx, m, n, *dev, 0)
    if n < 100000:  # and the tiles are the oracle's
        tiles, want = T.download(), oracle.csr2tile_row_major((m, n, rp, ci, v))
        for k in ("tile_ptr", "tile_columnidx", "tile_rowidx", "tile_nnz", "tile_csr_Ptr", "tile_csr_Value", "mask"):
            np.testing.assert_array_equal(tiles[k], want[k], err_msg=k)
        np.testing.assert_array_equal(tiles["tile_csr_Col"], want["tile_csr_Col"] & 15)
    if off_boundary:
        raw = torch.empty(16 * T.numtile + 1, dtype=torch.uint8, device=d)
        tiles = T.download()
        raw[1:] = torch.from_numpy(tiles["tile_csr_Ptr"]).to(d)
        owned, T.s.tile_csr_Ptr = T.s.tile_csr_Ptr, raw.data_ptr() + 1
    got = [x.cpu().numpy() for x in tsg.tiled_to_csr(ctx, T)]
    if off_boundary:
        T.s.tile_csr_Ptr = owned
    T.free()
    assert np.array_equal(got[0], rp)
    assert np.array_equal(got[1], ci)
    assert np.array_equal(got[2].view(np.uint64), v.view(np.uint64))


@pytest.mark.parametrize("m,n,tiles", [(16 * 300, 70, 255), (16 * 300, 70, 256), (16 * 300, 70, 257),
                                       (16 * 5000 + 3, 40, 4000), (16 * 262150, 33, 262149),
                                       (16 * 262150, 32000, 262149),
                                       (16 * 45000 + 3, 100, 40000)])
def test_column_view_of_columns_short_and_long(tsg, ctx, m, n, tiles):
    """Tile columns around the 256 tiles that a warp ranks, past them, and over
    more tile rows (262,144) than one bitmap pass, and few columns of many
    (sorted from 1,024 tiles a column on): tiles ascending by row in every column."""
    import torch
    rng = np.random.default_rng(tiles)
    rows = 16 * np.sort(rng.choice((m + 15) // 16, tiles, replace=False)).astype(np.int64)  # one entry a tile row
    cols = rng.integers(0, 16, tiles)
    extra = rng.integers(0, m, 2000)
    key = np.unique(np.concatenate([rows * n + cols, extra * n + rng.integers(16, n, 2000)]))
    r, ci = key // n, (key % n).astype(np.int32)
    rp = np.searchsorted(r, np.arange(m + 1)).astype(np.int32)
    d = torch.device("cuda", torch.cuda.current_device())
    T = tsg.csr_to_tiled(ctx, m, n, *[torch.from_numpy(x).to(d) for x in (rp, ci, rng.uniform(-1, 1, ci.size))],
                         tsg.TSG_TILED_CSC_VIEW)
    got = T.download(colmajor=True)
    T.free()
    tc = np.unique((ci // 16).astype(np.int64) * ((m + 15) // 16) + r // 16)  # (tile column, tile row)
    np.testing.assert_array_equal(got["csc_tile_rowidx"], tc % ((m + 15) // 16))
    np.testing.assert_array_equal(np.diff(got["csc_tile_ptr"]), np.bincount(tc // ((m + 15) // 16), minlength=(n + 15) // 16))


@pytest.mark.parametrize("flags", [0, 1, 2, 3])
def test_a_matrix_without_rows_needs_no_arrays(tsg, ctx, flags):
    import ctypes
    T = tsg.Tiled(ctx)
    tsg.check(tsg.lib().tsg_csr_to_tiled(ctx.handle, 0, 40, 0, None, None, None, flags, ctypes.byref(T.s)))
    got = [x.cpu().numpy() for x in tsg.tiled_to_csr(ctx, T)]
    assert T.numtile == 0 and np.array_equal(got[0], [0]) and got[1].size == 0
    T.free()
