"""Step 3 of products whose C tile rows hold few tiles (k_step3_nar), against
the oracle, bit for bit, at its edges: 4, 2 and 1 rows a task (16/17, 32/33
tiles), rows in chunks (64/65 tiles, tile columns 384 apart), rows left to the
SPA kernel (more than 128 tiles), a ragged last tile row, an A with no row
view, ranges of tile rows."""
import numpy as np
import pytest

from test_gpu_unstructured import _check, _same

pytestmark = pytest.mark.gpu

# (C tiles, their distance in tile columns) of a tile row
TILE_ROWS = [(1, 1), (3, 1), (16, 1), (17, 1), (32, 1), (33, 1), (64, 1), (65, 1), (130, 1), (3, 191), (3, 192), (3, 200),
             (16, 30), (17, 30), (64, 20)] + [(2, 1)] * 15


def _operands(seed):
    """Every tile row of A meets 64 rows of B of its own, whose columns lie in
    the tile row's tiles."""
    rng = np.random.default_rng(seed)
    n, B, A = 21000, [], []
    for I, (nt, s) in enumerate(TILE_ROWS):
        c0 = int(rng.integers(0, n // 16 - (nt - 1) * s))
        for _ in range(64):
            cols = (c0 + s * rng.integers(0, nt, 12)) * 16 + rng.integers(0, 16, 12)
            B.append(np.unique(cols[:rng.integers(0, 13)]))
        for r in range(16 if I + 1 < len(TILE_ROWS) else 5):
            A.append(np.sort(64 * I + rng.choice(64, rng.integers(0, 14), replace=False)))

    def csr(rows, cols):
        rp = np.concatenate([[0], np.cumsum([x.size for x in rows])]).astype(np.int32)
        ci = np.concatenate(rows).astype(np.int32)
        return len(rows), cols, rp, ci, rng.uniform(-1, 1, ci.size)

    return csr(A, len(B)), csr(B, n)


@pytest.mark.parametrize("seed", [1, 2])
@pytest.mark.parametrize("view", [True, False])
def test_narrow_rows(tsg, ctx, oracle, seed, view):
    A, B = _operands(seed)
    ctx.set_schedule("spa", dense=257)  # never the tile kernel
    try:
        info = _check(tsg, ctx, oracle, A, B, tsg.TSG_TILED_CSC_VIEW if view else tsg.TSG_TILED_PACKED_COL)
    finally:
        ctx.set_schedule("spa", dense=0)
    assert info["step3_name"] == "k_step3_nar"


def test_narrow_rows_without_the_fused_pass(tsg, ctx, oracle):
    """No row kinds: rows of more than 128 tiles are told by their tiles alone."""
    A, B = _operands(3)
    ctx.set_schedule("spa", dense=257)
    ctx.set_fusion(False)
    try:
        info = _check(tsg, ctx, oracle, A, B, tsg.TSG_TILED_CSC_VIEW)
    finally:
        ctx.set_fusion(True)
        ctx.set_schedule("spa", dense=0)
    assert info["step3_name"] == "k_step3_nar"


def test_narrow_rows_on_tile_row_ranges(tsg, ctx, oracle, gen):
    """The host call computes a band times a band in ranges of tile rows."""
    mat = gen.banded(120000, 5, seed=5)
    out = tsg.HostResultBuffers(mat[0], 1 << 22)
    ctx.set_schedule("spa", dense=257)
    try:
        got, info = tsg.spgemm_csr_host_overlap(ctx, mat, None, out)
    finally:
        ctx.set_schedule("spa", dense=0)
    assert info["nnz_C"] > 2 << 20  # more than one chunk
    assert info["step3_name"] == "k_step3_nar"
    _same(got[2:], oracle.gustavson(mat, mat, nthreads=8))
