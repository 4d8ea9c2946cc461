"""The pyramid's passes over two levels at once equal one pass a level
(test_gpu_preprocess.py checks that one against the oracle), byte for byte: sides
of no whole 4 rows or slices, odd ones, levels of one row, every voxel type, rows
of one chunk and of no whole chunk, and levels whose offsets rule a pass out."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [
    # dims, encoded bytes, channels, float, level alignment
    ((64, 64, 64), 1, 1, False, 256), ((64, 64, 64), 2, 1, False, 256), ((48, 50, 46), 1, 1, False, 256),
    ((48, 51, 37), 2, 1, False, 256), ((32, 40, 33), 2, 2, False, 256), ((32, 22, 45), 4, 1, True, 256),
    ((36, 30, 26), 4, 2, False, 256), ((20, 17, 19), 4, 4, False, 256), ((16, 9, 130), 1, 1, False, 256),
    ((8, 40, 7), 2, 1, False, 256), ((264, 6, 3), 2, 1, False, 256), ((40, 24, 24), 1, 1, False, 256),
    ((61, 40, 24), 1, 1, False, 256), ((64, 64, 64), 1, 1, False, 4), ((64, 64, 64), 1, 1, False, 1),
    ((64, 48, 40), 2, 1, False, 2), ((300, 200, 100), 2, 1, False, 256),
]


@pytest.mark.parametrize("dims,eb,ch,real,align", CASES)
def test_pyramid_equals_single_passes(gc, torch_cuda, dims, eb, ch, real, align):
    t = torch_cuda
    levels = [tuple(dims)]
    while min(levels[-1]) >= 2 and len(levels) < 8:
        levels.append(tuple(n // 2 for n in levels[-1]))
    layout = gc.Layout()
    layout.nb_levels = len(levels)
    offs, at = [], 0
    for l, d in enumerate(levels):
        for a in range(3):
            layout.mip[l][a] = layout.initial[l][a] = d[a]
        offs.append(at)
        at += -(-d[0] * d[1] * d[2] * eb // align) * align + (0 if align > 1 or l else 1)
    rng = np.random.default_rng(dims[0] + eb)
    n0 = dims[0] * dims[1] * dims[2] * eb
    raw = (rng.standard_normal(n0 // 4).astype(np.float32) * 1000).view(np.uint8) if real else \
        rng.integers(0, 256, n0, dtype=np.uint8)
    pyramid = t.full((at + 64,), 0xCD, dtype=t.uint8, device="cuda")
    pyramid[:n0].copy_(t.from_numpy(raw))
    single = pyramid.clone()
    gc.Mipmapper.process(pyramid.data_ptr(), layout, offs, eb, ch)
    for l in range(1, len(levels)):
        # one level at a time, through buffers of their own (aligned like a lone level)
        src = single[offs[l - 1]: offs[l - 1] + levels[l - 1][0] * levels[l - 1][1] * levels[l - 1][2] * eb].clone()
        dst = t.zeros(levels[l][0] * levels[l][1] * levels[l][2] * eb, dtype=t.uint8, device="cuda")
        gc.Mipmapper.down_scale(src.data_ptr(), dst.data_ptr(), levels[l - 1], eb, ch)
        single[offs[l]: offs[l] + dst.numel()].copy_(dst)
    t.cuda.synchronize()
    assert t.equal(pyramid, single)
