"""Film downloads: the threaded copy into pageable memory against the direct
copy into page-locked memory, its cost to the host while a render is still
running, and renders of other scenes beside it."""
import ctypes
import threading
import time

import numpy as np
import pytest
import torch

from vision_b200 import scenes

pytestmark = pytest.mark.gpu

PIXELS_1MB = (1 << 20) // 16  # of a linear film: the smallest threaded copy
CHUNK = (512 << 10) // 16
RING = 8 * CHUNK


def _scene(vb, ctx, width, height=1, seed=0):
    sc = scenes.box_room(width=width, height=height, max_depth=2, sampler='pcg')
    sc['sampler']['param']['seed'] = seed
    return vb.Scene(ctx, sc).build_accel()


def _download(vb, s, address, pixels, which=0):
    s.ctx.check(vb.lib.vs_film_download(s.handle, ctypes.c_void_p(address), pixels * 16, which), 'film_download')


@pytest.mark.parametrize('pixels', [PIXELS_1MB - 1, PIXELS_1MB, PIXELS_1MB + 1, 3 * CHUNK - 1, 3 * CHUNK + 1, RING - 1, RING,
                                    RING + 1, RING + CHUNK, RING + CHUNK + 1, 3 * RING + 5])
def test_threaded_copy_equals_direct_copy(vb, gpu_ctx, pixels):
    width = pixels if pixels < 1 << 16 else next(w for w in range(1 << 15, 0, -1) if pixels % w == 0)
    s = _scene(vb, gpu_ctx, width, pixels // width)
    s.render(0, 1)
    pinned = torch.empty(pixels * 4, dtype=torch.float32, pin_memory=True)
    _download(vb, s, pinned.data_ptr(), pixels)
    want = pinned.numpy().view(np.uint8)
    assert want.any()
    for misalign in (0, 1, 4):
        buf = np.full(pixels * 16 + 64, 0xa5, np.uint8)
        start = -buf.ctypes.data % 16 + misalign
        _download(vb, s, buf.ctypes.data + start, pixels)
        assert np.array_equal(buf[start:start + pixels * 16], want)
        assert np.all(buf[:start] == 0xa5) and np.all(buf[start + pixels * 16:] == 0xa5)  # nothing written around it


def test_download_behind_a_long_render_keeps_one_thread_busy(vb, gpu_ctx):
    s = _scene(vb, gpu_ctx, 1024, 1024)
    s.render(0, 1)
    s.film()
    s.render(0, 600)  # returns at once; hundreds of milliseconds of work
    cpu, wall = time.process_time(), time.perf_counter()
    s.film()
    cpu, wall = time.process_time() - cpu, time.perf_counter() - wall
    assert wall > 0.05
    # The waiting thread, and the copy itself at the end; not the helpers too.
    assert cpu < 1.7 * wall


def test_download_does_not_wait_for_a_later_render(vb, gpu_ctx):
    a, b = _scene(vb, gpu_ctx, 2048, 1024, 1), _scene(vb, gpu_ctx, 512, 512, 2)
    a.render(0, 1)
    want = a.film()
    b.render(0, 1500)
    gpu_ctx.check(vb.lib.vs_synchronize(b.handle), 'synchronize')
    t = time.perf_counter()
    b.render(0, 1500)
    gpu_ctx.check(vb.lib.vs_synchronize(b.handle), 'synchronize')
    later = time.perf_counter() - t
    a.render(0, 1)
    a.render(1, 40)  # the download waits for these
    got = []
    thread = threading.Thread(target=lambda: got.append((a.film(), time.perf_counter())))
    t = time.perf_counter()
    thread.start()
    time.sleep(0.01)
    b.render(0, 1500)
    queued = time.perf_counter() - t
    thread.join()
    gpu_ctx.check(vb.lib.vs_synchronize(b.handle), 'synchronize')
    assert got[0][0].shape == want.shape
    assert queued < 0.5 * later  # the render was queued while the download waited
    assert got[0][1] - t < 0.7 * later


def test_downloads_and_renders_on_several_threads(vb, gpu_ctx):
    made = [_scene(vb, gpu_ctx, 1200, 700, k) for k in range(3)]
    want = []
    for s in made:
        s.render(0, 2)
        want.append(s.film())
    wrong = []

    def work(k):
        for _ in range(12):
            made[k].render(0, 2)
            if not np.array_equal(made[k].film(), want[k]):
                wrong.append(k)
    threads = [threading.Thread(target=work, args=(k,)) for k in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def test_first_film_of_a_context_is_as_quick_as_the_next(vb, gpu_ctx):
    # The page-locked ring and its threads are the context's, made with it:
    # about 3 ms that the first film does not wait for.
    first, later = [], []
    for k in range(3):
        s = _scene(vb, vb.Context(0), 512, 512, k)
        s.render(0, 1)
        s.ctx.check(vb.lib.vs_synchronize(s.handle), 'synchronize')
        for times in (first, later, later):
            t = time.perf_counter()
            s.film()
            times.append(time.perf_counter() - t)
    assert min(first) < sorted(later)[3] + 1e-3
