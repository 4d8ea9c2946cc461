"""The ray caster's runs through one brick (no page walk between the samples of a
brick the ray surely stays in): frame by frame against the FP32 oracle, which
walks the page directory at every sample, bit for bit -- RGBA, t, colour state,
usage, requests and the rest of the cache state.

The cases are those where a run could leave its brick: boxes other than
[-1, 1]^3, view matrices that scale the ray directions, rays along the axes,
cameras inside the volume, bricks of every size, base steps shorter and longer
than the level's steps (empty bricks), and thin volumes."""
import numpy as np
import pytest

import scenario
from test_gpu_render import Scene

pytestmark = pytest.mark.gpu


def axis_camera(gc, axis, distance):
    eye = [0.0, 0.0, 0.0]
    eye[axis] = distance
    return gc.look_at(eye, up=(0.0, 0.0, 1.0) if axis == 1 else (0.0, 1.0, 0.0))


def scaled(m, s):
    return [x if k % 4 == 3 else x * s for k, x in enumerate(m)]


CASES = {
    # name: (size, bpc, B, c, camera, empty threshold, view arguments)
    "large_box": ((64, 64, 64), 1, 16, 1, lambda gc: scenario.orbit_camera(gc, 1, 12, 5.0), None,
                  dict(bbox_min=(-3.0, -1.5, -2.0), bbox_max=(2.5, 3.0, 3.0))),
    "small_box": ((64, 48, 64), 2, 16, 1, lambda gc: scenario.orbit_camera(gc, 2, 12, 1.2), None,
                  dict(bbox_min=(-0.3, -0.4, -0.25), bbox_max=(0.35, 0.3, 0.4), sampler=1)),
    "short_directions": ((64, 64, 64), 1, 16, 1, lambda gc: scaled(scenario.orbit_camera(gc, 1, 12, 2.4), 0.03), None,
                         dict()),
    "long_directions": ((64, 64, 64), 1, 16, 1, lambda gc: scaled(scenario.orbit_camera(gc, 1, 12, 2.4), 2.5), None,
                        dict()),
    "along_x": ((64, 64, 64), 1, 8, 1, lambda gc: axis_camera(gc, 0, 2.2), None, dict(focal=1e6)),
    "along_y": ((64, 64, 64), 2, 8, 2, lambda gc: axis_camera(gc, 1, -2.2), None, dict(focal=1e6, mode=1)),
    "along_z": ((64, 64, 64), 1, 16, 1, lambda gc: axis_camera(gc, 2, 30.0), None, dict(focal=30.0)),
    "inside": ((96, 64, 64), 2, 16, 1, lambda gc: gc.look_at((0.1, -0.2, 0.3), (0.9, 0.4, -0.6)), None,
               dict(focal=0.8)),
    "brick_4": ((32, 32, 32), 1, 4, 1, lambda gc: scenario.orbit_camera(gc, 4, 12, 2.6), None, dict()),
    "brick_64": ((96, 128, 96), 1, 64, 3, lambda gc: scenario.orbit_camera(gc, 5, 12, 2.6), None, dict()),
    "covering_0": ((64, 48, 64), 1, 16, 0, lambda gc: scenario.orbit_camera(gc, 4, 12, 2.4), None, dict()),
    "covering_0_tri": ((64, 48, 64), 2, 16, 0, lambda gc: scenario.orbit_camera(gc, 4, 12, 2.4), None, dict(sampler=1)),
    "thin": ((128, 24, 40), 1, 16, 1, lambda gc: scenario.orbit_camera(gc, 2, 12, 2.2), None, dict()),
    "empty_short_base": ((64, 64, 64), 1, 16, 1, lambda gc: scenario.orbit_camera(gc, 3, 12, 2.4), 24.0,
                         dict(tstep=0.003)),
    "empty_long_base": ((64, 64, 64), 1, 16, 1, lambda gc: scenario.orbit_camera(gc, 3, 12, 2.4), 24.0,
                        dict(tstep=0.11)),
}


@pytest.mark.parametrize("case", sorted(CASES))
def test_runs_match_the_walked_march(gc, orc, torch_cuda, case):
    size, bpc, B, c, cam, empty, kw = CASES[case]
    s = Scene(gc, orc, torch_cuda, size, bpc, B, c, (1, 1, 1), (8, 8, 8) if B < 64 else (3, 3, 3), 27)
    if empty is not None:
        d = scenario.gpu_volume(gc, torch_cuda, size, bpc, 21, 6)
        _, _, keys = gc.pre_process(s.vol, s.layout, d, empty_threshold=empty)
        assert keys
        s.cm.set_source_host(s.store, s.offs, keys)
        s.oc.set_source(s.ref, s.offs, keys)
    tf = scenario.bumps_tf(3)
    tf_dev = torch_cuda.from_numpy(tf.reshape(-1)).cuda()
    W, H = 45, 38
    g, o = s.buffers(W, H)
    v = s.view(cam(gc), W, H, tf_dev, 256, g, **dict(dict(early_alpha=0.99), **kw))
    converged, marched = False, 0
    for frame in range(60):
        s.cm.render(v)
        s.oc.render(v, tf, *o)
        torch_cuda.cuda.synchronize()
        tag = f"{case}, frame {frame}"
        assert np.array_equal(g[0].cpu().numpy().view(np.uint32), o[0].view(np.uint32)), tag
        assert np.array_equal(g[1].cpu().numpy(), o[1]), tag
        assert np.array_equal(g[2].cpu().numpy(), o[2]), tag
        converged = s.cm.update()
        assert converged == s.oc.update(), tag
        s.compare_cache(tag)
        if converged:
            break
    marched = s.cm.stats().rays_marched
    assert marched > 0 and s.cm.stats().bricks_installed > 0


@pytest.mark.parametrize("bpc,sampler", [(1, 0), (1, 1), (2, 0), (2, 1), (4, 1)])
def test_maximum_intensity_skips_change_nothing(gc, torch_cuda, bpc, sampler):
    """Bricks that cannot raise a ray's maximum are stepped through: image, t and
    maximum equal those without skipping, bit for bit, with values at both ends
    of the range (float voxels, which may lie outside [0, 1], are not skipped)."""
    t = torch_cuda
    n = 48
    gen = t.Generator().manual_seed(7)
    v = t.rand((n, n, n), generator=gen)
    v = t.where(v < 0.3, t.zeros(()), t.where(v > 0.98, t.ones(()), v * 0.9))  # bins 0 .. 63
    v[8:40, 8:40, 8:40] *= t.linspace(0.2, 1.0, 32)[:, None, None]
    if bpc == 4:
        d = (v * 3.0 - 1.0).reshape(-1).cuda()
    else:
        d = (v * (255 if bpc == 1 else 65535)).to(t.int32).to(t.uint8 if bpc == 1 else t.int16).reshape(-1).cuda()
    vol = gc.volume_desc((n, n, n), 8, 1, bpc)
    layout = gc.compute_layout(vol)
    store, offs, _ = gc.pre_process(vol, layout, d)
    tf = t.from_numpy(scenario.bumps_tf(3).reshape(-1)).cuda()
    images, samples = [], []
    for skip in (False, True):
        cm = gc.CacheManager(vol, layout, (10, 10, 10), max_requests=1000)
        cm.set_source_host(store, offs)
        W, H = 53, 41
        b = (t.zeros(W * H, dtype=t.int32, device="cuda"), t.zeros(W * H, device="cuda"),
             t.zeros(W * H * 4, device="cuda"))
        view = gc.make_view(scenario.orbit_camera(gc, 1, 12, 2.4), W, H, tf.data_ptr(), 256, b[0].data_ptr(),
                            b[1].data_ptr(), b[2].data_ptr(), mode=gc.MODE_MOP, sampler=sampler)
        gc.render_empty_skip(skip)
        try:
            for _ in range(60):
                cm.render(view)
                if cm.update():
                    break
            for x in b[1:]:
                x.zero_()
            before = cm.stats().samples
            cm.render(view)
            t.cuda.synchronize()
            samples.append(cm.stats().samples - before)
        finally:
            gc.render_empty_skip(True)
        images.append([x.cpu().numpy() for x in b])
        cm.close()
    for x, y in zip(*images):
        assert np.array_equal(x, y)
    assert images[0][2].any()
    assert samples[1] == samples[0] if bpc == 4 else samples[1] < samples[0]


@pytest.mark.parametrize("kind", ["u8", "u16", "f32", "two", "u8_two_level", "u8_b8"])
@pytest.mark.parametrize("mode,sampler", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_launches_of_few_and_many_rays_agree(gc, torch_cuda, kind, mode, sampler):
    """A launch of few rays takes more samples of a ray at a time than a launch of
    many, and a launch of one view holds its transfer function in shared memory:
    the same views in launches of one view, of one batch (over 24 x 32 rays per SM)
    and of one batch with two tables give the same image, t and colour state, bit
    for bit."""
    t = torch_cuda
    n, bpc, ch = 48, {"u16": 2, "f32": 4, "two": 2}.get(kind, 1), 2 if kind == "two" else 1
    B = 8 if kind == "u8_b8" else 16
    vol = gc.volume_desc((n, n, n), B, 1, bpc, ch)
    layout = gc.compute_layout(vol)
    if kind == "f32":
        d = scenario.gpu_volume(gc, t, (n, n, n), 1, 5, 6).float().div_(255.0)
    else:
        d = scenario.gpu_volume(gc, t, (n, n, n), bpc // ch, 5, 6, channels=ch)
    store, offs, _ = gc.pre_process(vol, layout, d)
    cm = gc.CacheManager(vol, layout, (9, 9, 9), max_requests=700, pt_block=4 if kind == "u8_two_level" else 0,
                         pt_slots=64 if kind == "u8_two_level" else 0)
    cm.set_source_host(store, offs)
    tf = scenario.tf2d(5) if ch == 2 else scenario.bumps_tf(3)
    tf_dev = t.from_numpy(tf.reshape(-1)).cuda()
    W, H, k = 181, 142, 8  # 8 views of 23 x 36 tiles
    bufs = [(t.zeros(W * H, dtype=t.int32, device="cuda"), t.zeros(W * H, device="cuda"),
             t.zeros(W * H * 4, device="cuda")) for _ in range(k)]
    views = [gc.make_view(scenario.orbit_camera(gc, i, 2 * k, 1.3 + 0.1 * i), W, H, tf_dev.data_ptr(), tf.shape[-2],
                          b[0].data_ptr(), b[1].data_ptr(), b[2].data_ptr(), focal=0.9, early_alpha=0.99, mode=mode,
                          sampler=sampler, tf_height=tf.shape[0] if ch == 2 else 0) for i, b in enumerate(bufs)]
    assert k * 23 * 36 > 24 * t.cuda.get_device_properties(0).multi_processor_count > 23 * 36
    for _ in range(100):
        cm.render_batch(views)
        if cm.update():
            break

    def images(render):
        for b in bufs:
            for x in b:
                x.zero_()
        render()
        t.cuda.synchronize()
        return [x.cpu().numpy() for b in bufs for x in b]

    one = images(lambda: [cm.render(v) for v in views])
    many = images(lambda: cm.render_batch(views))
    copy = tf_dev.clone()  # the views of this launch have different transfer functions
    for v in views[1::2]:
        v.tf = copy.data_ptr()
    mixed = images(lambda: cm.render_batch(views))
    assert any(x.any() for x in one)
    for x, y, z in zip(one, many, mixed):
        assert np.array_equal(x, y) and np.array_equal(x, z)

    # one view of many rays, alone and beside another view
    W, H = 640, 400
    assert W * H // 32 > 36 * t.cuda.get_device_properties(0).multi_processor_count
    bufs = [(t.zeros(W * H, dtype=t.int32, device="cuda"), t.zeros(W * H, device="cuda"),
             t.zeros(W * H * 4, device="cuda"))]
    large = gc.make_view(scenario.orbit_camera(gc, 3, 12, 1.4), W, H, tf_dev.data_ptr(), tf.shape[-2],
                         bufs[0][0].data_ptr(), bufs[0][1].data_ptr(), bufs[0][2].data_ptr(), focal=0.9,
                         early_alpha=0.99, mode=mode, sampler=sampler, tf_height=tf.shape[0] if ch == 2 else 0)
    for _ in range(100):
        cm.render(large)
        if cm.update():
            break
    alone = images(lambda: cm.render(large))
    beside = images(lambda: cm.render_batch([large, views[0]]))
    assert alone[0].any()
    for x, y in zip(alone, beside):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("width", [1, 2, 256, 512, 513])
def test_visible_bins_of_either_launch_agree(gc, torch_cuda, width):
    """A launch of one view holds its transfer function in shared memory and works
    out its visible value bins itself up to 512 entries, from there on (and for several views) a kernel
    before it does: bricks are skipped alike, so images, t, state and the number
    of samples are the same."""
    t = torch_cuda
    n = 48
    vol = gc.volume_desc((n, n, n), 8, 1, 1)
    layout = gc.compute_layout(vol)
    d = scenario.gpu_volume(gc, t, (n, n, n), 1, 9, 4)
    store, offs, _ = gc.pre_process(vol, layout, d)
    cm = gc.CacheManager(vol, layout, (11, 11, 11), max_requests=1000)
    cm.set_source_host(store, offs)
    table = scenario.bumps_tf(5, width)
    if width < 4:  # the bumps fall between so few entries
        table[:, 3] = 0.3
    tf = t.from_numpy(table.reshape(-1)).cuda()
    W, H = 60, 44
    b = (t.zeros(W * H, dtype=t.int32, device="cuda"), t.zeros(W * H, device="cuda"), t.zeros(W * H * 4, device="cuda"))
    view = gc.make_view(scenario.orbit_camera(gc, 2, 12, 2.4), W, H, tf.data_ptr(), width, b[0].data_ptr(),
                        b[1].data_ptr(), b[2].data_ptr())
    other = (t.zeros(1, dtype=t.int32, device="cuda"), t.zeros(1, device="cuda"), t.zeros(4, device="cuda"))
    beside = gc.make_view(gc.look_at((0.0, 0.0, 9.0), (0.0, 0.0, 20.0)), 1, 1, tf.data_ptr(), width,
                          other[0].data_ptr(), other[1].data_ptr(), other[2].data_ptr())  # looks away
    for _ in range(60):
        cm.render(view)
        if cm.update():
            break
    got = []
    for render in (lambda: cm.render(view), lambda: cm.render_batch([view, beside])):
        for x in b:
            x.zero_()
        before = cm.stats()
        render()
        t.cuda.synchronize()
        after = cm.stats()
        got.append([x.cpu().numpy() for x in b] + [after.samples - before.samples, after.rays_marched - before.rays_marched])
    for x, y in zip(*got):
        assert np.array_equal(x, y)
    assert got[0][3] > 0


@pytest.mark.parametrize("B,width,height,fewer", [(16, 64, 48, True), (8, 64, 64, True), (8, 33, 1, True), (16, 5, 7, True),
                                                  (16, 64, 65, False), (16, 600, 8, False), (4, 64, 48, False)])
@pytest.mark.parametrize("sampler", [0, 1])
def test_two_channel_skips_change_nothing(gc, torch_cuda, B, width, height, fewer, sampler):
    """Bricks of two 8-bit channels that the 2D transfer function cannot make
    visible are stepped through: image, t and state equal those without skipping,
    bit for bit; nothing is skipped with more than 64 table rows, tables too wide
    for shared memory, or brick rows of no whole 16 bytes."""
    t = torch_cuda
    n = 48
    z, y, x = np.meshgrid(*[np.linspace(-1, 1, n)] * 3, indexing="ij")
    rng = np.random.default_rng(2)
    c0 = np.clip(255 * np.exp(-3 * (x * x + y * y + z * z)) + rng.uniform(0, 8, (n, n, n)), 0, 255)
    c1 = np.clip(127 + 127 * np.sin(3 * x + 2 * y) + rng.uniform(-9, 9, (n, n, n)), 0, 255)
    d = t.from_numpy(np.stack([c0, c1], -1).astype(np.uint8).reshape(-1)).cuda()
    vol = gc.volume_desc((n, n, n), B, 1, 2, 2)
    layout = gc.compute_layout(vol)
    while tuple(layout.mip[layout.nb_levels - 1]) != tuple(layout.initial[layout.nb_levels - 1]):
        layout.nb_levels -= 1
    store, offs, _ = gc.pre_process(vol, layout, d)
    u, v = np.linspace(0, 1, width)[None, :], np.linspace(0, 1, height)[:, None]
    tf = np.zeros((height, width, 4), np.float32)
    tf[..., :3] = 0.5
    tf[..., 3] = np.where((u > 0.45) & (u < 0.8), 0.4, 0.0) * (1.0 if height < 4 else np.where(v > 0.4, 1.0, 0.0))
    tf_dev = t.from_numpy(tf.reshape(-1)).cuda()
    images, samples = [], []
    for skip in (False, True):
        cm = gc.CacheManager(vol, layout, (32, 32, 32), max_requests=4000)
        cm.set_source_host(store, offs)
        W, H = 57, 43
        b = (t.zeros(W * H, dtype=t.int32, device="cuda"), t.zeros(W * H, device="cuda"),
             t.zeros(W * H * 4, device="cuda"))
        view = gc.make_view(scenario.orbit_camera(gc, 1, 12, 2.4), W, H, tf_dev.data_ptr(), width, b[0].data_ptr(),
                            b[1].data_ptr(), b[2].data_ptr(), sampler=sampler, tf_height=height)
        gc.render_empty_skip(skip)
        try:
            for _ in range(200):
                cm.render(view)
                if cm.update():
                    break
            for a in b[1:]:
                a.zero_()
            before = cm.stats().samples
            cm.render(view)
            t.cuda.synchronize()
            samples.append(cm.stats().samples - before)
        finally:
            gc.render_empty_skip(True)
        images.append([a.cpu().numpy() for a in b])
        cm.close()
    for p, q in zip(*images):
        assert np.array_equal(p, q)
    assert images[0][0].any()
    assert samples[1] < samples[0] if fewer else samples[1] == samples[0]
