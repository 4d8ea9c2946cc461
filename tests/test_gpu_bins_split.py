"""Value bins of few and of many bricks: a block a brick below two bricks per SM (eight
for bricks above 8 KiB), a warp a brick from there on, one whole brick after the
other or out of big bricks.  Exact."""
import numpy as np
import pytest

from test_gpu_brick_bins import numpy_bins
from test_gpu_brick_scans import Geometry

pytestmark = pytest.mark.gpu


# 294 and 384, 512 bricks of level 0; the coarser levels have few
@pytest.mark.parametrize("size", [(98, 98, 84), (112, 112, 84), (112, 112, 112)])
@pytest.mark.parametrize("bb", [(1, 1, 1), (2, 2, 2), (3, 1, 2)])
@pytest.mark.parametrize("eb", [1, 2])
def test_few_and_many_bricks(gc, torch_cuda, size, bb, eb):
    t = torch_cuda
    g = Geometry(gc, size, 16, bb, eb)
    rng = np.random.default_rng(size[1] + bb[0] + eb)
    top = 255 if eb == 1 else 65535
    # every 512 values around a level of their own
    base = rng.integers(0, top, g.bytes // eb // 512)[:, None] + rng.integers(-top // 8, top // 8, (1, 512))
    store = np.ascontiguousarray(np.clip(base, 0, top).astype(np.uint8 if eb == 1 else np.uint16)).view(np.uint8).reshape(-1)
    dev = t.zeros(g.bytes, dtype=t.uint8, device="cuda")
    dev[: store.size].copy_(t.from_numpy(store))
    got = []
    for l in range(g.layout.nb_levels):
        nb = g.layout.nb_bricks[l]
        out = t.zeros(nb[0] * nb[1] * nb[2], dtype=t.int64, device="cuda")
        gc.brick_value_bins(g.vol, g.layout, l, dev.data_ptr() + g.offs[l], out.data_ptr())
        t.cuda.synchronize()
        got.append(out.cpu().numpy().view(np.uint64))
    assert np.array_equal(np.concatenate(got), numpy_bins(dev.cpu().numpy(), g.offs, g.vol, g.layout))


@pytest.mark.parametrize("size,bricks", [((168, 168, 112), 1152), ((168, 168, 154), 1584)])
def test_float_bricks_beside_the_line(gc, torch_cuda, size, bricks):
    t = torch_cuda
    g = Geometry(gc, size, 16, (1, 1, 1), 4)
    nb = g.layout.nb_bricks[0]
    assert nb[0] * nb[1] * nb[2] == bricks
    rng = np.random.default_rng(bricks)
    v = (rng.uniform(-0.3, 1.2, bricks)[:, None] + rng.uniform(-0.1, 0.1, (bricks, 4096))).astype(np.float32)
    v[:, ::97] = np.nan
    dev = t.from_numpy(v.reshape(-1)).cuda()
    out = t.zeros(bricks, dtype=t.int64, device="cuda")
    gc.brick_value_bins(g.vol, g.layout, 0, dev.data_ptr(), out.data_ptr())
    t.cuda.synchronize()
    lo, hi = np.nanmin(v, axis=1), np.nanmax(v, axis=1)
    b0 = np.clip(np.clip(np.floor(lo * np.float32(64)), 0, 63).astype(int) - 1, 0, 63)
    b1 = np.clip(np.clip(np.floor(hi * np.float32(64)), 0, 63).astype(int) + 1, 0, 63)
    want = [((1 << (int(q) + 1)) - 1) & ~((1 << int(p)) - 1) for p, q in zip(b0, b1)]
    assert out.cpu().numpy().view(np.uint64).tolist() == want
