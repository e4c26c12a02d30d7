"""The chain on rows of every length mod 4. fy_gpu_restore_u8 keeps the deconvolved volume and the
guided pairs in rows padded to 4 voxels, staged by tensor copies; the stages called one by one on dense
rows stage ragged ones 4 bytes at a time. A voxel's sums take the same taps in the same order either
way, and the pairs turn into coefficients by the same expressions, so the tolerance is none."""
import ctypes as C

import numpy as np
import pytest

from tests.test_gpu_restore import cfg_for, phys

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [65, 66, 67, 68])         # two tiles of 64 columns, the second nearly empty
@pytest.mark.parametrize("radius,win", [(1, 3), (2, 5), (3, 7), (4, 9), (1, 9), (3, 5)])
def test_rows(gpu, nx, radius, win):
    import torch
    lib, ph, shape = gpu.load(), phys(gpu), (21, 35, nx)
    rng = np.random.default_rng(nx + radius)
    ramp = np.linspace(60, 190, nx)[None, None, :] + rng.standard_normal(shape) * 6
    u8 = torch.from_numpy(np.clip(np.rint(ramp), 0, 255).astype(np.uint8)).cuda()
    got, dec, want = (torch.empty(shape, dtype=torch.float32, device="cuda") for _ in range(3))
    scratch = torch.empty(lib.fy_gpu_noise_scratch_bytes(*shape), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    at = lambda t: C.c_void_p(t.data_ptr())
    cfg = cfg_for(gpu, None)
    cfg.guided_radius, cfg.noise_win = radius, win
    assert lib.fy_gpu_restore_u8(at(u8), at(got), *shape, 0.0, 1.0, C.byref(ph), C.byref(cfg), None) == 0
    assert lib.fy_gpu_deconvolve_ex(at(u8), 1, 0.0, 1.0, at(dec), *shape, C.byref(ph), 0.05, 1, 1.0, None) == 0
    assert lib.fy_gpu_estimate_noise(at(dec), *shape, win, 10.0, 0.4, at(scratch), None) == 0
    nm = gpu.NoiseModel()
    assert lib.fy_gpu_noise_model(at(scratch), *shape, C.byref(nm), None) == 0
    eps = lib.fy_guided_eps_for_noise(nm.noise_ref)
    assert lib.fy_gpu_guided(at(dec), at(want), *shape, radius, eps, 1, None) == 0
    torch.cuda.synchronize()
    assert np.array_equal(got.cpu().numpy(), want.cpu().numpy())
