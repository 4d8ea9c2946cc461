"""Levels of odd rows around the size from which they are down-sampled through
16-byte windows (eight bytes out a thread): rows of one chunk and more, just below
the line, on it and above, equal a torch reduction."""
import numpy as np
import pytest

from test_gpu_mip_rows import reduced

pytestmark = pytest.mark.gpu


def check(gc, t, rng, dims, eb, ch, real=False):
    n = dims[0] * dims[1] * dims[2] * eb
    host = (rng.standard_normal(n // 4) * 9).astype(np.float32).view(np.uint8) if real else \
        rng.integers(0, 256, n, dtype=np.uint8)
    src = t.from_numpy(host).cuda()
    out = (dims[0] // 2) * (dims[1] // 2) * (dims[2] // 2) * eb
    dst = t.full((out + 16,), 0xEE, dtype=t.uint8, device="cuda")
    gc.Mipmapper.down_scale(src.data_ptr(), dst.data_ptr(), dims, eb, ch)
    t.cuda.synchronize()
    assert t.equal(dst[:out], reduced(t, src, dims, eb, ch, real)), dims
    assert bool((dst[out:] == 0xEE).all()), dims


@pytest.mark.parametrize("eb,ch", [(1, 1), (2, 1), (4, 2)])
def test_short_rows_above_the_line(gc, torch_cuda, eb, ch):
    rng = np.random.default_rng(eb + ch)
    for X in list(range(2, 36)) + [61, 127]:  # 360 x 151 rows out: above the line from one chunk a row on
        check(gc, torch_cuda, rng, (X, 720, 303), eb, ch)


@pytest.mark.parametrize("eb,ch,real", [(1, 1, False), (2, 1, False), (4, 2, False), (2, 2, False), (4, 4, False),
                                        (4, 1, True)])
def test_sizes_beside_the_line(gc, torch_cuda, eb, ch, real):
    rng = np.random.default_rng(7 * eb + ch)
    line = 28672 if eb == ch and ch > 1 else 53248
    for X in (3, 9, 17, 33, 67):
        chunks = (X // 2 * eb + 7) // 8
        for rows in (line // (chunks * 64) - 1, line // (chunks * 64), line // (chunks * 64) + 1):
            check(gc, torch_cuda, rng, (X, 2 * rows + 1, 128), eb, ch, real)
