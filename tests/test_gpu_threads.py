"""Contexts on two host threads at once: products whose step 2 of wide rows
takes different amounts of shared memory, launched side by side."""
import threading

import numpy as np
import pytest

from test_gpu_unstructured import _rows, _tiled

pytestmark = pytest.mark.gpu


def test_products_of_different_widths_on_two_threads(tsg, oracle):
    import torch
    A = _rows(40, 120, [6] * 40, 1)
    errors, done = [], []
    start = threading.Barrier(2)

    def work(n):
        try:
            torch.cuda.set_device(0)
            ctx = tsg.Context(0, own_stream=True)
            B = _rows(120, n, [8] * 120, n)
            want = oracle.gustavson(A, B)
            tA, tB = (_tiled(tsg, ctx, x, tsg.TSG_TILED_CSC_VIEW) for x in (A, B))
            torch.cuda.synchronize()
            start.wait()
            for _ in range(400):
                C, info = tsg.spgemm(ctx, tA, tB)
                assert info["nnz_C"] == want[3].size
                C.free()
            C, _ = tsg.spgemm(ctx, tA, tB)
            got = [x.cpu().numpy() for x in tsg.tiled_to_csr(ctx, C)]
            assert np.array_equal(got[1], want[3]) and np.array_equal(got[2].view(np.uint64), want[4].view(np.uint64))
            for t in (C, tA, tB):
                t.free()
            ctx.close()
            done.append(n)
        except Exception as e:  # noqa: BLE001 - reported below
            errors.append((n, e))

    threads = [threading.Thread(target=work, args=(n,)) for n in (98304, 12000)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    assert len(done) == 2
