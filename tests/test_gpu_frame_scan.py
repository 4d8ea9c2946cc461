"""The frame's scans -- request scan, used-slot counts and the LRU partition -- at
the edges of their tiles (8192 request entries, 1024 to 16,384 slots): one entry or slot
more or less than a whole number of tiles, flags at the first and last entries of
a tile, none, all, and more than the list holds.  Lists, totals and LRU order
equal a numpy restatement."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def geometry(gc, n):
    """A one-level layout of n bricks along x."""
    vol = gc.volume_desc((16, 16, 16), 16, 1, 1)
    layout = gc.compute_layout(vol)
    assert layout.nb_levels == 1
    layout.nb_bricks[0][0], layout.nb_bricks[0][1], layout.nb_bricks[0][2] = n, 1, 1
    return layout


@pytest.mark.parametrize("n", [2, 3, 5, 255, 8191, 8192, 8193, 8194, 16385, 16386, 16388, 40961, 70003])
@pytest.mark.parametrize("maxreq", [1, 50, 9000])
def test_miss_list_at_tile_edges(gc, torch_cuda, n, maxreq):
    t = torch_cuda
    rng = np.random.default_rng(n + maxreq)
    layout = geometry(gc, n)
    edges = [i for i in (0, 1, 3, 4, 127, 128, 1023, 1024, 8191, 8192, 8193, n - 3, n - 2, n - 1) if 0 <= i < n]
    for flagged in ([], edges, sorted(rng.choice(n, max(1, n // 3), replace=False)), range(n)):
        req = rng.integers(0, 7, n).astype(np.int32)
        req[list(flagged)] = 7
        want = np.nonzero(req[: n - 1] == 7)[0]  # the scan's range ends before the last entry
        d = t.from_numpy(req).cuda()
        out = t.full((maxreq * 4,), -1, dtype=t.int32, device="cuda")
        total = t.full((1,), -1, dtype=t.int32, device="cuda")
        gc.miss_list_noalloc(d.data_ptr(), n, 7, layout, maxreq, out.data_ptr(), total.data_ptr())
        t.cuda.synchronize()
        assert int(total.item()) == want.size
        got = out.cpu().numpy().reshape(-1, 4)
        k = min(maxreq, want.size)
        assert np.array_equal(got[:k, 0], want[:k]) and not got[:k, 1:].any()
        assert (got[k:] == -1).all()


# one cluster of up to eight blocks (1024, 2048, ... 16,384 slots each, 131,072 in all) and
# the count + partition kernels above
@pytest.mark.parametrize("slots", [(1, 1, 1), (31, 1, 1), (4095, 1, 1), (16, 16, 16), (4097, 1, 1), (64, 64, 3), (1024, 1, 1), (1025, 1, 1), (64, 64, 2), (8193, 1, 1), (16385, 1, 1),
                                   (128, 128, 1), (128, 64, 5), (128, 128, 8), (131073, 1, 1),
                                   (64, 64, 64), (262145, 1, 1), (270000, 1, 1)])
def test_lru_order_at_tile_edges(gc, torch_cuda, slots):
    B = 16 if slots[0] * slots[1] * slots[2] < 20000 else 4
    vol = gc.volume_desc((64, 64, 64), B, 1, 1)
    layout = gc.compute_layout(vol)
    cm = gc.CacheManager(vol, layout, slots, max_requests=1)
    cm.set_source_callback(lambda *a: gc.BRICK_UNKNOWN)
    n = slots[0] * slots[1] * slots[2]
    rng = np.random.default_rng(n)
    order = np.arange(n)
    for share in (0.0, 0.3, 1.0, 0.01):
        ts = cm.timestamp()
        usage = np.where(rng.random(n) < share, ts, max(0, ts - 1)).astype(np.uint32)
        if share == 0.01:
            usage[[0, n - 1]] = ts
        cm.load_buffer(gc.DUMP_USAGE, usage)
        cm.update()
        used = usage[order] == ts
        order = np.concatenate([order[used], order[~used]])
        lru = np.zeros(n, dtype=np.dtype([("c", np.uint32, 3), ("level", np.uint32), ("v", np.float32, 3)]))
        cm.dump(gc.DUMP_LRU, lru)
        sx, sy = slots[0], slots[1]
        want = np.stack([(order % sx) * B, (order // sx % sy) * B, (order // (sx * sy)) * B], 1)
        assert np.array_equal(lru["c"], want), share
        assert cm.stats().last_used == used.sum()
    assert cm.stats().device_error == 0
