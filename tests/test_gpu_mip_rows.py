"""Down-sampling of levels whose rows start at any byte equals a torch reduction:
every alignment of source and output rows, last chunks of every length, levels of
a few bytes (loads that would pass the level's end), every voxel type, and a
destination off its voxels' grid (the value-by-value kernel, as for small levels)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def reduced(t, raw, dims, eb, ch, real):
    X, Y, Z = dims
    cb = eb // ch
    if real:
        a = raw.view(t.float32).double().reshape(Z, Y, X, 1)
    else:
        a = raw.view(t.uint8 if cb == 1 else t.int16).to(t.int32).reshape(Z, Y, X, ch)
        a = a & (0xFF if cb == 1 else 0xFFFF)
    a = a[: Z // 2 * 2, : Y // 2 * 2, : X // 2 * 2].reshape(Z // 2, 2, Y // 2, 2, X // 2, 2, ch)
    if real:  # the order of the sum: x, y, z
        s = t.zeros((Z // 2, Y // 2, X // 2, 1), dtype=t.float64, device=raw.device)
        for dz in range(2):
            for dy in range(2):
                for dx in range(2):
                    s = s + a[:, dz, :, dy, :, dx]
        return (s / 8.0).float().reshape(-1).view(t.uint8)
    s = a.sum(dim=(1, 3, 5)) // 8
    return (s.to(t.uint8) if cb == 1 else s.to(t.int16)).reshape(-1).view(t.uint8)


@pytest.mark.parametrize("eb,ch,real", [(1, 1, False), (2, 1, False), (2, 2, False), (4, 2, False), (4, 4, False),
                                        (4, 1, True), (3, 3, False)])
@pytest.mark.parametrize("yz", [(3, 7), (300, 303)])  # below and above the size that takes windows
def test_rows_of_any_length(gc, torch_cuda, eb, ch, real, yz):
    t = torch_cuda
    rng = np.random.default_rng(eb * 10 + yz[0])
    for X in list(range(2, 36)) + [61, 127]:
        dims = (X, *yz)
        n = X * yz[0] * yz[1] * eb
        host = (rng.standard_normal(n // 4) * 9).astype(np.float32).view(np.uint8) if real else \
            rng.integers(0, 256, n, dtype=np.uint8)
        src = t.from_numpy(host).cuda()
        out = (X // 2) * (yz[0] // 2) * (yz[1] // 2) * eb
        for shift in (0, eb, 1):
            if shift == 1 and eb != 1 and eb != 3:
                continue  # voxels are stored whole
            dst = t.full((out + 16,), 0xEE, dtype=t.uint8, device="cuda")
            gc.Mipmapper.down_scale(src.data_ptr(), dst.data_ptr() + shift, dims, eb, ch)
            t.cuda.synchronize()
            assert t.equal(dst[shift: shift + out], reduced(t, src, dims, eb, ch, real)), (X, shift)
            assert bool((dst[:shift] == 0xEE).all()) and bool((dst[shift + out:] == 0xEE).all()), (X, shift)
