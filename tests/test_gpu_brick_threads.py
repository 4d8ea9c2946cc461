"""Bricking from several host threads at once: shapes whose slabs need different
amounts of shared memory above the default limit launch side by side, and every
call's bricks equal those of the same call made alone."""
import threading

import pytest

pytestmark = pytest.mark.gpu


def test_threads_with_different_slab_sizes(gc, torch_cuda):
    t = torch_cuda
    # slabs of 73,728 (64^3 bricks) and 139,264 bytes (128^3), of 4-byte voxels
    work = []
    for B, size in ((64, (64, 64, 64)), (128, (128, 128, 128)), (64, (100, 64, 64)), (128, (150, 128, 128))):
        vol = gc.volume_desc(size, B, 1, 4, 1)
        layout = gc.compute_layout(vol)
        nbig = list(layout.nb_big_bricks[0])
        level = t.randint(0, 2**31 - 1, (size[0] * size[1] * size[2],), dtype=t.int32, device="cuda")
        want = t.zeros(nbig[0] * nbig[1] * nbig[2] * B**3, dtype=t.int32, device="cuda")
        gc.process_bricking(level.data_ptr(), size, vol, nbig, want.data_ptr())
        work.append((vol, nbig, size, level, want))
    t.cuda.synchronize()
    errors, wrong = [], []
    start = threading.Barrier(len(work))

    def run(vol, nbig, size, level, want):
        stream = t.cuda.Stream()
        got = t.zeros_like(want)
        t.cuda.synchronize()
        start.wait()
        try:
            for _ in range(1500):
                gc.process_bricking(level.data_ptr(), size, vol, nbig, got.data_ptr(), stream.cuda_stream)
        except gc.GcError as e:
            errors.append(str(e))
        stream.synchronize()
        if not t.equal(got, want):
            wrong.append(size)

    threads = [threading.Thread(target=run, args=w) for w in work]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not errors, errors
    assert not wrong, wrong
