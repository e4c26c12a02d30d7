"""Host deconvolutions through the staged copies: sizes at the edges of the chunks (1 MB) and of the pinned
ring (16 MB), in place, from pinned memory and from several threads at once. The device form on the same
input is the reference; the copies move bytes, so the tolerance is none."""
import ctypes as C
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(64, 64, 63), (64, 64, 64), (65, 64, 64), (2, 1024, 1031), (64, 256, 257), (128, 256, 129)]


def _device(gpu, vol, ph):
    import torch
    d = torch.from_numpy(vol).cuda()
    out = torch.empty_like(d)
    torch.cuda.synchronize()
    assert gpu.load().fy_gpu_deconvolve_ex(C.c_void_p(d.data_ptr()), 0, 0.0, 0.0, C.c_void_p(out.data_ptr()), *vol.shape,
                                           C.byref(ph), 0.015, 0, 1.0, None) == 0
    torch.cuda.synchronize()
    return out.cpu().numpy()


@pytest.mark.parametrize("shape", SHAPES)
def test_staged_copies(gpu, shape):
    import torch
    ph, lib = gpu.physics(), gpu.load()
    vol = np.random.default_rng(shape[2]).uniform(0, 1, shape).astype(np.float32)
    want = _device(gpu, vol, ph)
    assert np.array_equal(gpu.deconvolve(vol, ph, 0.015), want)
    buf = vol.copy()
    assert lib.fy_deconvolve(buf.ctypes.data, buf.ctypes.data, *shape, C.byref(ph), 0.015) == 0
    assert np.array_equal(buf, want)
    pin = torch.from_numpy(vol).pin_memory()
    out = np.empty_like(vol)
    assert lib.fy_deconvolve(pin.data_ptr(), out.ctypes.data, *shape, C.byref(ph), 0.015) == 0
    assert np.array_equal(out, want)


def test_many_callers(gpu):
    """More callers than the helper allowance serves."""
    ph = gpu.physics()
    vols = [np.random.default_rng(i).uniform(0, 1, (40 + i, 128, 128)).astype(np.float32) for i in range(12)]
    want = [_device(gpu, v, ph) for v in vols]
    bad = []

    def work(i):
        for _ in range(3):
            if not np.array_equal(gpu.deconvolve(vols[i], ph, 0.015), want[i]):
                bad.append(i)
        gpu.load().fy_gpu_release()

    th = [threading.Thread(target=work, args=(i,)) for i in range(len(vols))]
    for t in th:
        t.start()
    for t in th:
        t.join(120)
    assert not bad and not any(t.is_alive() for t in th)
