"""The level bricker's blocks of 64, 128 and 256 threads: slabs of so many bricks of 4^3,
8^3 and 16^3 voxels that their output chunks or their copies just fit two a thread,
just do not, or leave a last slab of another size; few and many slices a block.
Bytes equal the numpy restatement."""
import numpy as np
import pytest

from test_gpu_brick_slabs import numpy_bricks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,eb,ch", [(4, 2, 1), (4, 4, 1), (4, 8, 4), (6, 8, 4), (8, 1, 1), (8, 2, 1), (8, 4, 1), (8, 3, 3),
                                     (16, 1, 1), (16, 2, 1)])
@pytest.mark.parametrize("c", [0, 1])
@pytest.mark.parametrize("bb", [(1, 1, 1), (2, 2, 1)])
def test_slabs_of_every_size(gc, torch_cuda, B, eb, ch, c, bb):
    t = torch_cuda
    rng = np.random.default_rng(B * 100 + eb * 10 + c)
    beff = B - 2 * c
    for bricks in (1, 2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 34, 63, 64, 65, 66):
        # (a level of `bricks` along x, of a few in y and of one to several slices in z)
        dims = (bricks * beff - (1 if bricks % 3 else 0), 2 * beff + 1, beff + bricks % 5)
        dims = tuple(max(1, d) for d in dims)
        vol = gc.volume_desc(tuple(max(d, B) for d in dims), B, c, eb, ch, bb)
        nb = [-(-d // beff) for d in dims]
        nbig = [-(-n // b) for n, b in zip(nb, bb)]
        raw = rng.integers(0, 256, dims[0] * dims[1] * dims[2] * eb, dtype=np.uint8)
        dev = t.from_numpy(raw).cuda()
        want = numpy_bricks(raw, dims, eb, B, c, bb, nbig)
        out = t.full((want.size + 16,), 0xEE, dtype=t.uint8, device="cuda")
        gc.process_bricking(dev.data_ptr(), dims, vol, nbig, out.data_ptr())
        t.cuda.synchronize()
        got = out.cpu().numpy()
        assert np.array_equal(got[: want.size], want), bricks
        assert (got[want.size:] == 0xEE).all(), bricks
