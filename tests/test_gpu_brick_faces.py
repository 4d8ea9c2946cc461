"""Rays along the faces between bricks, a few roundings to either side of them: the
brick a sample's page walk finds and the brick its voxel lies in can differ there.
Frame by frame against the FP32 oracle, bit for bit: RGBA, t, colour state and the
cache state."""
import numpy as np
import pytest

import scenario
from test_gpu_brick_runs import axis_camera
from test_gpu_render import Scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bpc,B,c,mode,sampler", [(1, 16, 1, 0, 0), (1, 16, 2, 0, 1), (2, 16, 1, 1, 1), (2, 32, 1, 0, 1),
                                                  (1, 32, 3, 1, 0), (1, 8, 1, 0, 1)])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_rays_along_faces(gc, orc, torch_cuda, axis, bpc, B, c, mode, sampler):
    n = 80
    s = Scene(gc, orc, torch_cuda, (n, n, n), bpc, B, c, (1, 1, 1), (10, 10, 10), 27)
    tf = scenario.bumps_tf(3)
    tf_dev = torch_cuda.from_numpy(tf.reshape(-1)).cuda()
    beff = B - 2 * c
    real = -(-n // beff) * beff
    for k in (1, real // beff // 2):
        face = np.float64(k) * beff / n  # normalized position of the k-th face: position * n / real * bricks = k
        for ulps in (-3, -2, -1, 0, 1, 2, 3):
            m = list(axis_camera(gc, axis, 2.2))
            for a in range(3):
                if a != axis:
                    p = face if a < 2 else 1.0 - face  # z is flipped
                    x = np.float32((p - 0.495) / 0.495)
                    m[4 * a + 3] = float(x + np.float32(ulps) * np.spacing(x))
            W = H = 5
            g, o = s.buffers(W, H)
            v = s.view(m, W, H, tf_dev, 256, g, early_alpha=0.99, focal=1e6, mode=mode, sampler=sampler)
            for frame in range(30):
                s.cm.render(v)
                s.oc.render(v, tf, *o)
                torch_cuda.cuda.synchronize()
                tag = f"face {k}, {ulps} ulps, frame {frame}"
                assert np.array_equal(g[0].cpu().numpy().view(np.uint32), o[0].view(np.uint32)), tag
                assert np.array_equal(g[1].cpu().numpy(), o[1]), tag
                assert np.array_equal(g[2].cpu().numpy(), o[2]), tag
                converged = s.cm.update()
                assert converged == s.oc.update(), tag
                s.compare_cache(tag)
                if converged:
                    break
    assert s.cm.stats().samples > 0
