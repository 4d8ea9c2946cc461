"""The kernels that scan a store of bricks 16 bytes at a time (value bins, empty
flags) at the edges of what they accept: bricks below and above one warp's share,
rows of one and of several chunks, brick sizes that are no power of two, big
bricks, stores off the 16-byte grid (the value-by-value kernels), and for the
flags values at the threshold, NaNs and several channels.  Exact."""
import numpy as np
import pytest

from test_gpu_brick_bins import numpy_bins

pytestmark = pytest.mark.gpu


class Geometry:
    """One level of bricks as the value bins take it."""

    def __init__(self, gc, size, B, bb, eb):
        self.vol = gc.volume_desc(size, B, 1, eb, 1, bb)
        self.layout = gc.compute_layout(self.vol)
        offs, self.bytes, self.big = gc.brick_store_offsets(self.layout, self.vol)
        self.offs = offs


@pytest.mark.parametrize("size,B,bb,eb,shift", [
    ((60, 40, 30), 16, (1, 1, 1), 1, 0), ((60, 40, 30), 16, (1, 1, 1), 2, 0), ((70, 70, 40), 32, (1, 1, 1), 2, 0),
    ((90, 40, 60), 24, (1, 1, 1), 2, 0), ((90, 40, 60), 24, (2, 1, 3), 2, 0), ((50, 40, 40), 8, (1, 1, 1), 2, 0),
    ((64, 30, 40), 16, (2, 2, 2), 1, 0), ((70, 70, 70), 32, (1, 2, 1), 1, 0), ((60, 40, 30), 16, (1, 1, 1), 2, 8),
    ((50, 40, 40), 8, (1, 1, 2), 1, 0), ((64, 64, 64), 64, (1, 1, 1), 1, 0)])
def test_value_bins_match_numpy(gc, torch_cuda, size, B, bb, eb, shift):
    t = torch_cuda
    g = Geometry(gc, size, B, bb, eb)
    rng = np.random.default_rng(B * 10 + eb)
    # each big brick around a level of its own, so that the ranges differ
    n = g.bytes // g.big
    top = 255 if eb == 1 else 65535
    base = rng.integers(0, top, n)[:, None] + rng.integers(-top // 8, top // 8, (n, g.big // eb))
    store = np.ascontiguousarray(np.clip(base, 0, top).astype(np.uint8 if eb == 1 else np.uint16)).view(np.uint8).reshape(-1)
    dev = t.zeros(g.bytes + 16, dtype=t.uint8, device="cuda")
    dev[shift:shift + g.bytes].copy_(t.from_numpy(store))
    got = []
    for l in range(g.layout.nb_levels):
        nb = g.layout.nb_bricks[l]
        out = t.zeros(nb[0] * nb[1] * nb[2], dtype=t.int64, device="cuda")
        gc.brick_value_bins(g.vol, g.layout, l, dev.data_ptr() + shift + g.offs[l], out.data_ptr())
        t.cuda.synchronize()
        got.append(out.cpu().numpy().view(np.uint64))
    assert np.array_equal(np.concatenate(got), numpy_bins(store, g.offs, g.vol, g.layout))


@pytest.mark.parametrize("eb", [4])
def test_value_bins_of_floats(gc, torch_cuda, eb):
    """Float voxels below, inside and above [0, 1], with NaNs among them."""
    t = torch_cuda
    g = Geometry(gc, (32, 32, 32), 16, (1, 1, 1), eb)
    rng = np.random.default_rng(3)
    n = g.bytes // g.big
    v = (rng.uniform(-0.3, 1.2, n)[:, None] + rng.uniform(-0.1, 0.1, (n, g.big // 4))).astype(np.float32)
    v[:, ::97] = np.nan
    dev = t.from_numpy(v.reshape(-1)).cuda()
    nb = g.layout.nb_bricks[0]
    k = nb[0] * nb[1] * nb[2]
    out = t.zeros(k, dtype=t.int64, device="cuda")
    gc.brick_value_bins(g.vol, g.layout, 0, dev.data_ptr() + g.offs[0], out.data_ptr())
    t.cuda.synchronize()
    lo, hi = np.nanmin(v[:k], axis=1), np.nanmax(v[:k], axis=1)
    b0 = np.clip(np.clip(np.floor(lo * np.float32(64)), 0, 63).astype(int) - 1, 0, 63)
    b1 = np.clip(np.clip(np.floor(hi * np.float32(64)), 0, 63).astype(int) + 1, 0, 63)
    want = [((1 << (int(q) + 1)) - 1) & ~((1 << int(p)) - 1) for p, q in zip(b0, b1)]
    assert out.cpu().numpy().view(np.uint64).tolist() == want


@pytest.mark.parametrize("cb,ch,B,bb,shift", [(1, 1, 16, (1, 1, 1), 0), (2, 1, 16, (1, 1, 1), 0), (1, 2, 16, (2, 2, 2), 0),
                                              (2, 1, 32, (1, 1, 1), 0), (4, 1, 16, (1, 1, 1), 0), (4, 1, 32, (1, 1, 1), 0),
                                              (2, 1, 5, (1, 1, 1), 0), (1, 1, 4, (1, 1, 1), 0), (2, 1, 16, (1, 1, 1), 6),
                                              (1, 3, 16, (1, 1, 1), 0)])
def test_empty_flags_match_numpy(gc, torch_cuda, cb, ch, B, bb, shift):
    t = torch_cuda
    vol = gc.volume_desc((64, 64, 64), B, 1, cb * ch, ch, bb)
    values = B ** 3 * bb[0] * bb[1] * bb[2] * ch
    n, threshold = 41, 30.0
    rng = np.random.default_rng(cb * 100 + B)
    a = rng.integers(0, 30, (n, values)).astype({1: np.uint8, 2: np.uint16, 4: np.float32}[cb])
    for i, at in enumerate((0, values - 1, values // 2, values // 3, 17)):  # one value at the threshold
        a[3 * i + 1, at] = 30
    if cb == 4:
        a[20, 5] = np.nan
        a[21, values - 1] = np.inf
        a[22, :] = -np.inf
    a[30] = 200
    raw = a.reshape(-1).view(np.uint8)
    dev = t.zeros(raw.size + 16, dtype=t.uint8, device="cuda")
    dev[shift:shift + raw.size].copy_(t.from_numpy(raw))
    flags = t.full((n,), 7, dtype=t.uint8, device="cuda")
    gc.process_empty(dev.data_ptr() + shift, n, vol, threshold, flags.data_ptr())
    t.cuda.synchronize()
    want = (a < np.float32(threshold)).all(axis=1).astype(np.uint8)
    assert want.any() and not want.all()
    assert np.array_equal(flags.cpu().numpy(), want)
