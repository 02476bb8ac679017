"""Exclusive scans through the conversion's tile counts, at the scan's edges:
a block of 8,192 items and one more, up to 1,024 blocks whose sums every block
adds up itself, and past them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("items", [1, 7, 8191, 8192, 8193, 16384, 3 * 8192 + 5, 1024 * 8192, 1024 * 8192 + 1])
def test_scan_of_tile_counts(tsg, ctx, items):
    """One row of A a tile row, 0 to 3 tiles: tile_ptr is the scan of their counts."""
    import torch
    d = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=d)
    g.manual_seed(items)
    counts = torch.randint(0, 4, (items,), device=d, generator=g)
    m = 16 * items
    rp = torch.zeros(m + 1, dtype=torch.int64, device=d)
    per = torch.zeros(items, 16, dtype=torch.int64, device=d)
    per[:, 3] = counts
    rp[1:] = torch.cumsum(per.flatten(), 0)
    nnz = int(rp[-1])
    at = torch.arange(nnz, device=d) - torch.repeat_interleave(torch.cumsum(counts, 0) - counts, counts)
    T = tsg.csr_to_tiled(ctx, m, 64, rp.to(torch.int32), (16 * at).to(torch.int32),
                         torch.ones(nnz, dtype=torch.float64, device=d), 0)
    got = T.download()["tile_ptr"]
    T.free()
    np.testing.assert_array_equal(got, np.concatenate([[0], np.cumsum(counts.cpu().numpy())]))
