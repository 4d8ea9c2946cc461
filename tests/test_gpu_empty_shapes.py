"""Empty flags of large big bricks in every split over warps and blocks (a warp a big
brick; a block for one and for several, whose first bytes it looks at first):
a single value at the threshold anywhere in a big brick makes it non-empty."""
import pytest

pytestmark = pytest.mark.gpu


# bytes of a big brick: 32 KiB (B 32), 128 KiB, 256 KiB; numbers around one block per
# big brick, several, and a warp each
@pytest.mark.parametrize("cb,B,n", [(1, 32, 1), (1, 32, 608), (1, 32, 609), (1, 32, 1217), (1, 32, 2433), (1, 32, 7295), (1, 32, 7297), (2, 32, 2433),
                                    (4, 32, 41), (4, 32, 2433), (1, 64, 2433), (2, 40, 2431)])
def test_one_value_anywhere(gc, torch_cuda, cb, B, n):
    t = torch_cuda
    vol = gc.volume_desc((128, 128, 128), B, 1, cb, 1)
    values = B ** 3
    kind = {1: t.uint8, 2: t.int16, 4: t.float32}[cb]
    a = t.full((n, values), 29, dtype=kind, device="cuda")
    per = 16 // cb  # values of a chunk
    places = [0, per - 1, per, 32 * per - 1, 32 * per, 128 * per - 1, 128 * per, 1024 * per - 1, 1024 * per,
              values // 2 + 1, values - per, values - 1]
    want = t.ones(n, dtype=t.uint8, device="cuda")
    for k, at in enumerate(places):
        a[2 * k::2 * len(places), min(at, values - 1)] = 30  # every other big brick
        want[2 * k::2 * len(places)] = 0
    if cb == 4 and n > 30:
        a[1, values - 1] = float("nan")
        a[3, 5] = float("inf")
        a[5] = float("-inf")
        want[1] = want[3] = 0
    flags = t.full((n + 8,), 7, dtype=t.uint8, device="cuda")
    gc.process_empty(a.data_ptr(), n, vol, 30.0, flags.data_ptr())
    t.cuda.synchronize()
    assert t.equal(flags[:n], want)
    assert bool((flags[n:] == 7).all())
