"""The visible value bins of two-channel views, worked out by a launch before the ray
caster's: tables from one entry to the widest, and launches with different tables
one after the other on one stream."""
import numpy as np
import pytest

import scenario
from test_gpu_brick_runs import test_two_channel_skips_change_nothing as skips_change_nothing

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,width,height", [(16, 512, 64), (16, 300, 63), (8, 512, 2), (16, 97, 31)])
@pytest.mark.parametrize("sampler", [0, 1])
def test_tables_of_any_size(gc, torch_cuda, B, width, height, sampler):
    skips_change_nothing(gc, torch_cuda, B, width, height, True, sampler)


def test_launches_with_different_tables(gc, torch_cuda):
    t = torch_cuda
    n = 48
    rng = np.random.default_rng(4)
    z, y, x = np.meshgrid(*[np.linspace(-1, 1, n)] * 3, indexing="ij")
    c0 = 255 * np.exp(-3 * (x * x + y * y + z * z)) * rng.uniform(0.9, 1, (n, n, n))
    d = t.from_numpy(np.stack([c0, 120 + 100 * x], -1).astype(np.uint8).reshape(-1)).cuda()
    vol = gc.volume_desc((n, n, n), 16, 1, 2, 2)
    layout = gc.compute_layout(vol)
    while tuple(layout.mip[layout.nb_levels - 1]) != tuple(layout.initial[layout.nb_levels - 1]):
        layout.nb_levels -= 1
    store, offs, _ = gc.pre_process(vol, layout, d)
    cm = gc.CacheManager(vol, layout, (16, 16, 16), max_requests=4000)
    cm.set_source_host(store, offs)
    W, H = 40, 30
    views, bufs, keep = [], [], []
    for k in range(3):  # each table shows another band of channel 0
        u = np.linspace(0, 1, 64)[None, :].repeat(16, 0)
        tf = np.zeros((16, 64, 4), np.float32)
        tf[..., k] = 1.0
        tf[..., 3] = np.where((u > 0.1 + 0.3 * k) & (u < 0.3 + 0.3 * k), 0.5, 0.0)
        keep.append(t.from_numpy(tf.reshape(-1)).cuda())
        for _ in range(50):  # 150 views, more than the rows kept
            b = (t.zeros(W * H, dtype=t.int32, device="cuda"), t.zeros(W * H, device="cuda"),
                 t.zeros(W * H * 4, device="cuda"))
            bufs.append(b)
            views.append((k, gc.make_view(scenario.orbit_camera(gc, 1, 12, 2.4), W, H, keep[-1].data_ptr(), 64,
                                          b[0].data_ptr(), b[1].data_ptr(), b[2].data_ptr(), tf_height=16)))
    for k in range(3):
        for _ in range(100):
            cm.render(views[50 * k][1])
            if cm.update():
                break
    for b in bufs:
        b[1].zero_()
        b[2].zero_()
    t.cuda.synchronize()
    for i in rng.permutation(len(views)):  # launches one after the other, tables mixed
        cm.render(views[i][1])
    t.cuda.synchronize()
    images = [b[0].cpu().numpy() for b in bufs]
    gc.render_empty_skip(False)
    try:
        for k in range(3):
            for a in bufs[50 * k][1:]:
                a.zero_()
            cm.render(views[50 * k][1])
            t.cuda.synchronize()
            want = bufs[50 * k][0].cpu().numpy()
            assert want.any()
            for i in range(50 * k, 50 * k + 50):
                assert np.array_equal(images[i], want), (k, i)
    finally:
        gc.render_empty_skip(True)
    cm.close()
