"""The level bricker at the edges of its slabs: rows of any length (so that every
row starts at its own byte of a 16-byte chunk), levels smaller than a brick, brick
rows of 8 bytes, of one and of many chunks and of no power of two, coverings wider
than a brick's inner part, several channels, big bricks, more bricks than the
level needs, and more slabs than blocks.  Bytes equal a numpy restatement of the
bricking rule (process_bricking, Bricker_v2.cpp:79-252): brick b holds voxels
[b (B - 2c) - c, b (B - 2c) - c + B) per axis, zeros outside the level, and is zero
when its start b (B - 2c) lies outside the level on some axis."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [
    # dims, encoded bytes, channels, B, c, big brick
    ((61, 35, 29), 1, 1, 16, 1, (1, 1, 1)),
    ((61, 35, 29), 2, 1, 16, 1, (1, 1, 1)),
    ((333, 20, 17), 1, 1, 16, 1, (1, 1, 1)),
    ((515, 30, 16), 2, 1, 16, 2, (1, 1, 1)),
    ((64, 64, 64), 2, 1, 16, 0, (1, 1, 1)),
    ((5, 3, 2), 1, 1, 16, 1, (1, 1, 1)),
    ((1, 40, 7), 2, 1, 16, 1, (1, 1, 1)),
    ((45, 33, 20), 1, 1, 8, 1, (1, 1, 1)),
    ((45, 33, 20), 1, 1, 8, 3, (2, 1, 2)),
    ((70, 30, 20), 2, 1, 24, 1, (1, 1, 1)),
    ((70, 30, 20), 1, 1, 24, 11, (1, 1, 1)),
    ((50, 40, 30), 2, 1, 16, 7, (1, 1, 1)),
    ((47, 31, 18), 3, 3, 16, 1, (1, 1, 1)),
    ((47, 31, 18), 8, 4, 16, 1, (1, 2, 1)),
    ((49, 35, 21), 4, 1, 16, 1, (2, 2, 2)),
    ((75, 66, 40), 1, 1, 32, 1, (1, 1, 1)),
    ((75, 66, 40), 2, 1, 32, 3, (2, 1, 1)),
    ((140, 130, 20), 1, 1, 64, 1, (1, 1, 1)),
    ((150, 130, 20), 2, 1, 128, 1, (1, 1, 1)),
    ((70, 20, 10), 8, 4, 128, 1, (1, 1, 1)),
    ((41, 30, 20), 1, 1, 9, 1, (1, 1, 1)),
    ((41, 30, 20), 2, 2, 4, 1, (1, 1, 1)),
]


def numpy_bricks(raw, dims, eb, B, c, bb, nbig):
    beff = B - 2 * c
    nb = [n * b for n, b in zip(nbig, bb)]
    level = raw.reshape(dims[2], dims[1], dims[0], eb)
    grid = np.zeros([n * B for n in nb[::-1]] + [eb], np.uint8)
    padded = np.zeros([(n - 1) * beff + B + d + 2 * c for n, d in zip(nb[::-1], dims[::-1])] + [eb], np.uint8)
    padded[c:c + dims[2], c:c + dims[1], c:c + dims[0]] = level
    for z in range(nb[2]):
        for y in range(nb[1]):
            for x in range(nb[0]):
                if x * beff < dims[0] and y * beff < dims[1] and z * beff < dims[2]:
                    grid[z * B:z * B + B, y * B:y * B + B, x * B:x * B + B] = \
                        padded[z * beff:z * beff + B, y * beff:y * beff + B, x * beff:x * beff + B]
    bv = [b * B for b in bb]
    grid = grid.reshape(nbig[2], bv[2], nbig[1], bv[1], nbig[0], bv[0], eb)
    return np.ascontiguousarray(grid.transpose(0, 2, 4, 1, 3, 5, 6)).reshape(-1)


@pytest.mark.parametrize("dims,eb,ch,B,c,bb", CASES)
@pytest.mark.parametrize("shift", [0, 2])  # a level off the 16-byte grid takes the voxel bricker
def test_bricks_match_numpy(gc, torch_cuda, dims, eb, ch, B, c, bb, shift):
    t = torch_cuda
    if shift and eb == 8:
        shift = 8
    if shift and eb == 4:
        shift = 4
    vol = gc.volume_desc(dims, B, c, eb, ch, bb)
    beff = B - 2 * c
    nbig = [-(-(-(-d // beff)) // b) + (1 if i == 0 else 0) for i, (d, b) in enumerate(zip(dims, bb))]
    rng = np.random.default_rng(dims[0] + 31 * B + eb)
    n = dims[0] * dims[1] * dims[2] * eb
    raw = rng.integers(1, 256, n, dtype=np.uint8)
    ref = numpy_bricks(raw, dims, eb, B, c, bb, nbig)
    dev = t.zeros(n + 16, dtype=t.uint8, device="cuda")
    dev[shift:shift + n].copy_(t.from_numpy(raw))
    out = t.full((ref.size,), 0xAB, dtype=t.uint8, device="cuda")
    gc.process_bricking(dev.data_ptr() + shift, dims, vol, nbig, out.data_ptr())
    t.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), ref)
