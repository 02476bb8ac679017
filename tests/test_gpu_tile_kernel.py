"""The tile kernel's two forms (a lane per C column for A tiles of 64 values and
more on average, a lane per C row below), chosen per product, against the
oracle, bit for bit: around the limit, with full, nearly empty and mixed A
tiles, ragged edges, and both forms in one batch."""
import numpy as np
import pytest

from test_gpu_unstructured import _check, _same, _tiled

pytestmark = pytest.mark.gpu


def _blocks(nt, counts, seed, n=None):
    """Tile-tridiagonal matrix, counts[i] values in the tiles of tile row i."""
    rng = np.random.default_rng(seed)
    n = n or 16 * nt
    at = set()
    for I in range(nt):
        for J in range(max(0, I - 1), min(nt, I + 2)):
            for q in rng.choice(256, counts[I % len(counts)], replace=False):
                r, c = 16 * I + int(q) // 16, 16 * J + int(q) % 16
                if r < n and c < n:
                    at.add((r, c))
    r, c = (np.array(x, np.int64) for x in zip(*sorted(at)))
    return n, n, np.searchsorted(r, np.arange(n + 1)).astype(np.int32), c.astype(np.int32), rng.uniform(-1, 1, r.size)


CASES = [((63,), None), ((64,), None), ((65,), None), ((256,), None), ((1,), None), ((24,), 101), ((120,), 101),
         ((2, 256, 9), None), ((1, 180, 1), 97)]


@pytest.mark.parametrize("counts,n", CASES)
@pytest.mark.parametrize("sched,dense", [("tiles", 0), ("spa", 1)])
def test_both_forms_of_the_tile_kernel(tsg, ctx, oracle, counts, n, sched, dense):
    A, B = _blocks(7, counts, 1, n), _blocks(7, (30, 90), 2, n)
    ctx.set_schedule(sched, dense=dense)
    try:
        info = _check(tsg, ctx, oracle, A, B, tsg.TSG_TILED_CSC_VIEW)
    finally:
        ctx.set_schedule("spa", dense=0)
    T = len({(r // 16, c // 16) for r in range(A[0]) for c in A[3][A[2][r]:A[2][r + 1]]})
    assert info["step3_name"] == ("k_step3" if A[3].size >= 64 * T else "k_step3_tile_rows")


@pytest.mark.parametrize("sets", [CASES, CASES[4:6], CASES[1:4]])
@pytest.mark.parametrize("sched", ["tiles", "spa"])
def test_both_forms_in_one_batch(tsg, ctx, oracle, sets, sched):
    mats = [(_blocks(7, c, 1, n), _blocks(7, (30, 90), 2, n)) for c, n in sets]
    pairs = [tuple(_tiled(tsg, ctx, x, tsg.TSG_TILED_CSC_VIEW) for x in ab) for ab in mats]
    batch = tsg.Batch(ctx, pairs, sched, dense=1 if sched == "spa" else 0)
    for _ in range(2):
        batch.run()
        batch.sync()
        for p, (a, b) in enumerate(mats):
            _same([x.cpu().numpy() for x in tsg.tiled_to_csr(ctx, batch.product(p))], oracle.gustavson(a, b))
    batch.close()
