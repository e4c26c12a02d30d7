"""The host deconvolutions on buffers that are not plain host memory. Under unified addressing the
copies take device, managed and pinned addresses as well, below and above the sizes from which plain
host memory is staged (4 MB); the bytes are the same, so the tolerance is none."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(64, 64, 63), (64, 64, 64), (90, 128, 257)])
@pytest.mark.parametrize("src", ["host", "pinned", "device"])
@pytest.mark.parametrize("dst", ["host", "pinned", "device"])
def test_buffers(gpu, src, dst, shape):
    import torch
    lib, ph = gpu.load(), gpu.physics()
    vol = np.random.default_rng(shape[2]).uniform(0, 1, shape).astype(np.float32)
    want = gpu.deconvolve(vol, ph, 0.015)
    put = {"host": lambda t: t, "pinned": lambda t: t.pin_memory(), "device": lambda t: t.cuda()}
    a, b = put[src](torch.from_numpy(vol)), put[dst](torch.zeros(shape))
    torch.cuda.synchronize()
    for f, param in ((lib.fy_deconvolve, 0.015), (lib.fy_deconvolve_matched, 0.05)):
        assert f(a.data_ptr(), b.data_ptr(), *shape, C.byref(ph), param) == 0
        if f is lib.fy_deconvolve:
            assert np.array_equal(b.cpu().numpy(), want)
