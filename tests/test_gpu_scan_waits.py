"""The bounded waits of the request scan run out where a predecessor publishes
nothing (GC_TEST_NOALLOC_SILENT_TILE): a flagged tile of the same group of 256
tiles, and one of a later group that waits for the whole group.  The call then
reports GC_MISS_LIST_FAILED, and the next call gives the right list."""
import time

import numpy as np
import pytest

from test_gpu_frame_scan import geometry

pytestmark = pytest.mark.gpu

TILE = 8192


@pytest.mark.parametrize("silent,tiles,flagged", [(0, 3, 2), (1, 4, 3), (5, 300, 299)])
def test_a_flagged_tile_waits_and_gives_up(gc, torch_cuda, monkeypatch, silent, tiles, flagged):
    t = torch_cuda
    n = tiles * TILE + 1
    assert flagged > silent and flagged * TILE < n - 1  # a later tile has to wait for the silent one
    layout = geometry(gc, n)
    req = t.zeros(n, dtype=t.int32, device="cuda")
    req[flagged * TILE: flagged * TILE + 5] = 7
    out = t.full((50 * 4,), -1, dtype=t.int32, device="cuda")
    total = t.full((1,), -1, dtype=t.int32, device="cuda")

    def call():
        gc.miss_list_noalloc(req.data_ptr(), n, 7, layout, 50, out.data_ptr(), total.data_ptr())
        t.cuda.synchronize()
        return int(total.item()) & 0xFFFFFFFF

    assert call() == 5
    monkeypatch.setenv("GC_TEST_NOALLOC_SILENT_TILE", str(silent))
    begin = time.perf_counter()
    assert call() == gc.MISS_LIST_FAILED
    # 2^22 polls of a word in the L2 take far more than this; a scan without a wait, microseconds
    assert time.perf_counter() - begin > 0.05
    monkeypatch.delenv("GC_TEST_NOALLOC_SILENT_TILE")
    out.fill_(-1)
    assert call() == 5
    got = out.cpu().numpy().reshape(-1, 4)
    assert np.array_equal(got[:5, 0], flagged * TILE + np.arange(5)) and (got[5:] == -1).all()
