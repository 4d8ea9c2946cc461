"""The scans whose tiles read their predecessors' counts by groups of 256 tiles: the
request scan (8192 entries a tile) and the LRU partition (4096 slots a tile) at
the edges of a group, with flags nowhere, at the edges, once a tile and
everywhere.  Lists, totals and LRU order equal a numpy restatement."""
import numpy as np
import pytest

from test_gpu_frame_scan import geometry

pytestmark = pytest.mark.gpu

SCAN_TILE, LRU_TILE, GROUP = 8192, 4096, 256
LRU_GROUPED = 12288  # tiles above which the LRU partition sums groups


@pytest.mark.parametrize("tiles,more", [(255, 0), (256, 0), (256, 1), (257, 0), (512, 0), (513, 1), (700, 77), (1024, 0)])
def test_miss_list_at_group_edges(gc, torch_cuda, tiles, more):
    t = torch_cuda
    n = tiles * SCAN_TILE + more + 1  # the scan's range ends before the last entry
    layout = geometry(gc, n)
    rng = np.random.default_rng(tiles)
    edge = GROUP * SCAN_TILE
    edges = [i for i in (0, edge - 1, edge, edge + 1, 2 * edge - 1, 2 * edge, n - 2, n - 1) if i < n]
    maxreq = 9000
    out = t.empty(maxreq * 4, dtype=t.int32, device="cuda")
    total = t.empty(1, dtype=t.int32, device="cuda")
    every = np.arange(0, n, SCAN_TILE)
    for flagged in ([], edges, every + rng.integers(0, SCAN_TILE, every.size), every[every >= n - 3 * SCAN_TILE], None):
        req = rng.integers(0, 7, n).astype(np.int32)
        if flagged is None:
            req[:] = 7
        else:
            req[[i for i in flagged if i < n]] = 7
        want = np.nonzero(req[: n - 1] == 7)[0]
        d = t.from_numpy(req).cuda()
        for _ in range(2):  # the first call leaves the scratch as the second expects it
            out.fill_(-1)
            total.fill_(-1)
            gc.miss_list_noalloc(d.data_ptr(), n, 7, layout, maxreq, out.data_ptr(), total.data_ptr())
            t.cuda.synchronize()
            assert int(total.item()) == want.size
            got = out.cpu().numpy().reshape(-1, 4)
            k = min(maxreq, want.size)
            assert np.array_equal(got[:k, 0], want[:k]) and not got[:k, 1:].any()
            assert (got[k:] == -1).all()


@pytest.mark.parametrize("n", [GROUP * LRU_TILE + 1, LRU_GROUPED * LRU_TILE, LRU_GROUPED * LRU_TILE + 1,
                               (LRU_GROUPED + GROUP) * LRU_TILE + 5])
def test_lru_order_at_group_edges(gc, torch_cuda, n):
    vol = gc.volume_desc((64, 64, 64), 4, 1, 1)
    layout = gc.compute_layout(vol)
    cm = gc.CacheManager(vol, layout, (n, 1, 1), max_requests=1)  # 64 bytes a slot
    cm.set_source_callback(lambda *a: gc.BRICK_UNKNOWN)
    rng = np.random.default_rng(n)
    order = np.arange(n)
    for share in (0.3, 0.001):
        ts = cm.timestamp()
        usage = np.where(rng.random(n) < share, ts, max(0, ts - 1)).astype(np.uint32)
        usage[[0, n - 1]] = ts
        cm.load_buffer(gc.DUMP_USAGE, usage)
        cm.update()
        used = usage[order] == ts
        order = np.concatenate([order[used], order[~used]])
        lru = np.zeros(n, dtype=np.dtype([("c", np.uint32, 3), ("level", np.uint32), ("v", np.float32, 3)]))
        cm.dump(gc.DUMP_LRU, lru)
        assert np.array_equal(lru["c"][:, 0], order * 4), share
        assert not lru["c"][:, 1:].any()
        assert cm.stats().last_used == used.sum()
    assert cm.stats().device_error == 0
    cm.close()


@pytest.mark.parametrize("n", [131073, 131074, 131075, 131076, 2490368, 2490371])
def test_used_slots_of_any_remainder(gc, torch_cuda, n):
    """The used slots of pools above one cluster, counted four at a time."""
    vol = gc.volume_desc((64, 64, 64), 4, 1, 1)
    cm = gc.CacheManager(vol, gc.compute_layout(vol), (n, 1, 1), max_requests=1)
    cm.set_source_callback(lambda *a: gc.BRICK_UNKNOWN)
    rng = np.random.default_rng(n)
    for used in ([], [0], [n - 1], [n - 2, n - 3], rng.choice(n, 1000, replace=False), np.arange(n)):
        ts = cm.timestamp()
        usage = np.full(n, ts + 1, np.uint32)
        usage[np.asarray(used, np.int64)] = ts
        cm.load_buffer(gc.DUMP_USAGE, usage)
        cm.update()
        assert cm.stats().last_used == len(used)
    assert cm.stats().device_error == 0
    cm.close()
