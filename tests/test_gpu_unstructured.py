"""The dense tile kernel against the oracle: bands on both sides of the dense
path, ragged tiles, infinite and NaN values.  Values bit for bit: the order of
the sums is the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


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
