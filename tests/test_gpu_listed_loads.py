"""Loads that the device resolves from the miss list itself (one-brick big bricks,
no empty bricks, host stores and device pyramids) leave the cache as the general
route does: two caches fed the same usage and request buffers, one of them with a
callback source over the same bricks, hold the same page directory, LRU order,
pool, miss lists and counters after every update -- also when the buffer flags
entries of the directory's padding (no brick there: the general route takes the
list and counts a load error), lists one brick and more than it has room for."""
import ctypes

import numpy as np
import pytest

import scenario

pytestmark = pytest.mark.gpu


class Store:
    """A volume's bricks in host memory and its pyramid on the device."""

    def __init__(self, gc, torch, size, B, bpc, seed):
        self.vol = gc.volume_desc(size, B, 1, bpc)
        self.layout = gc.compute_layout(self.vol)
        d = scenario.gpu_volume(gc, torch, size, bpc, seed, 5)
        self.host, self.offs, _ = gc.pre_process(self.vol, self.layout, d, pin=True)
        self.poffs, total = gc.pyramid_offsets(self.layout, bpc)
        self.pyramid = torch.zeros(total, dtype=torch.uint8, device="cuda")
        self.pyramid[: d.numel()].copy_(d)
        gc.Mipmapper.process(self.pyramid.data_ptr(), self.layout, self.poffs, bpc, 1)
        torch.cuda.synchronize()
        self.big = B ** 3 * bpc

    def callback(self, gc):
        def load(user, level, x, y, z, dst, nbytes):
            nb = self.layout.nb_big_bricks[level]
            if x >= nb[0] or y >= nb[1] or z >= nb[2]:
                return gc.BRICK_UNKNOWN
            at = self.offs[level] + ((z * nb[1] + y) * nb[0] + x) * self.big
            ctypes.memmove(dst, self.host.data_ptr() + at, nbytes)
            return gc.BRICK_SUCCESS

        return load

    def give(self, gc, cm, kind, volume):
        if kind == "host":
            cm.set_source_host(self.host, self.offs, volume=volume)
        elif kind == "device":
            cm.set_source_device(self.pyramid.data_ptr(), self.poffs, volume=volume, keep=self.pyramid)
        else:
            cm.set_source_callback(self.callback(gc), volume=volume)


@pytest.mark.parametrize("kinds,B,bpcs,maxreq,pt", [
    (("host",), 16, (1,), 40, 0), (("device",), 16, (2,), 40, 0), (("host",), 8, (2,), 1, 0),
    (("device",), 8, (1,), 90, 4), (("host", "device"), 16, (1, 2), 40, 0), (("device", "host"), 8, (2, 1), 64, 2)])
def test_listed_loads_equal_the_general_route(gc, torch_cuda, kinds, B, bpcs, maxreq, pt):
    t = torch_cuda
    stores = [Store(gc, t, (64 - 8 * i, 48, 40 + 8 * i), B, bpc, 3 + i) for i, bpc in enumerate(bpcs)]
    caches = []
    for general in (False, True):
        shared = [(s.vol, s.layout) for s in stores] if len(stores) > 1 else None
        cm = gc.CacheManager(stores[0].vol, stores[0].layout, (5, 5, 4), max_requests=maxreq, shared=shared,
                             pt_block=pt, pt_slots=6 if pt else 0)
        for i, (s, k) in enumerate(zip(stores, kinds)):
            s.give(gc, cm, "callback" if general else k, i)
        caches.append(cm)
    a, b = caches
    n = a.info.mrpd_dims[0] * a.info.mrpd_dims[1] * a.info.mrpd_dims[2]
    rng = np.random.default_rng(B + maxreq)
    slot = B ** 3 * max(bpcs)
    for frame in range(12):
        ts = a.timestamp()
        assert ts == b.timestamp()
        req = rng.integers(0, max(1, ts), n).astype(np.uint32)
        req[rng.integers(0, n, (0, 1, maxreq, 3 * maxreq)[frame % 4])] = ts  # padding entries among them
        usage = np.where(rng.random(100) < 0.4, ts, 0).astype(np.uint32)
        got = []
        for cm in caches:
            cm.load_buffer(gc.DUMP_REQUESTS, req)
            cm.load_buffer(gc.DUMP_USAGE, usage)
            conv = cm.update()
            state = [conv]
            for what, size, dt in ((gc.DUMP_MRPD, 4 * n, np.uint32), (gc.DUMP_LRU, 7 * 100, np.uint32),
                                   (gc.DUMP_POOL, 100 * slot, np.uint8)):
                x = np.zeros(size, dt)
                cm.dump(what, x)
                state.append(x)
            st = cm.stats()
            total, misses = cm.last_misses()
            state += [misses, total, st.requests_served, st.bricks_installed, st.bricks_empty, st.load_errors,
                      st.device_error]
            got.append(state)
        for x, y in zip(*got):
            assert np.array_equal(x, y), frame
    assert a.stats().bricks_installed > 0
