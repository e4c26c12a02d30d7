"""Z scales of the deconvolution's frequencies for which its weight table has no scale: refused with
FY_EINVAL by every entry point before it does anything (so without a device too), and large finite
ones, which crowd the rows into few cells of the table and reach its last one.

Tolerance against the FP64 oracle: as tests/test_gpu_regfft.py derives it, a transform of P points
rounds at most log2(P) times per direction (2^-24 each), on values of at most 1 times the largest
weight of the kind (8, or 1/(2 sqrt(0.05)) for the matched filter)."""
import ctypes as C
import math

import numpy as np
import pytest

import oracle

INF, NAN = math.inf, math.nan
# kind, sigma_z, fz2_scale; 1e200 squared overflows, 1e-310 leaves 4096 / umax above the doubles
BAD = [(2, 0.0, NAN), (2, 0.0, INF), (1, INF, 1.0), (1, 1e200, 1.0)]


def _phys(fy, sigma_z=0.0):
    return fy.physics(psf_sigma_vox=1.0, psf_sigma_z_vox=sigma_z)


def _buffers(shape):
    return np.zeros(shape, np.float32), np.zeros(shape, np.float32)


@pytest.mark.parametrize("shape", [(64, 40, 64), (10, 12, 14), (640, 3, 5)])
@pytest.mark.parametrize("kind,sigma_z,scale", BAD)
def test_refused(fy, kind, sigma_z, scale, shape):
    lib, ph, (a, b) = fy.load(), _phys(fy, sigma_z), _buffers(shape)
    u8 = np.zeros(shape, np.uint8)
    assert lib.fy_gpu_deconvolve_ex(a.ctypes.data, 0, 0.0, 1.0, b.ctypes.data, *shape, C.byref(ph), 0.05, kind, scale,
                                    None) == fy.FY_EINVAL
    if kind == 1:
        assert lib.fy_deconvolve_matched(a.ctypes.data, b.ctypes.data, *shape, C.byref(ph), 0.05) == fy.FY_EINVAL
    cfg = fy.RestoreCfg()
    lib.fy_restore_cfg_default(C.byref(cfg))
    cfg.deconv_kind, cfg.fz2_scale = kind, scale
    assert lib.fy_gpu_restore_u8(u8.ctypes.data, b.ctypes.data, *shape, 0.0, 1.0, C.byref(ph), C.byref(cfg),
                                 None) == fy.FY_EINVAL
    item = fy.BatchCube(u8.ctypes.data, b.ctypes.data, *shape, 0.0, 1.0, ph)
    assert lib.fy_gpu_restore_u8_batch(C.byref(item), 1, C.byref(cfg), None) == fy.FY_EINVAL


def test_no_table_scale(fy):
    """Only z is longer than one voxel, and its scale is a denormal: 4096 / umax is infinite."""
    a, b = _buffers((64, 1, 1))
    assert fy.load().fy_gpu_deconvolve_ex(a.ctypes.data, 0, 0.0, 1.0, b.ctypes.data, 64, 1, 1, C.byref(_phys(fy)), 0.05,
                                          2, 1e-310, None) == fy.FY_EINVAL


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(64, 40, 64), (10, 12, 14), (640, 3, 5), (256, 5, 7), (1, 1, 1)])
@pytest.mark.parametrize("kind,sigma_z,scale", [(2, 0.0, 1e6), (1, 1e3, 1.0), (2, 0.0, 1e300), (2, 0.0, 1e-300)])
def test_large_finite_scale(gpu, kind, sigma_z, scale, shape):
    import torch
    lib, ph = gpu.load(), _phys(gpu, sigma_z)
    v = np.random.default_rng(sum(shape)).random(shape, dtype=np.float32)
    p = math.prod(lib.fy_next_fft_size(d) for d in shape)
    rph = oracle.RefPhysics(*[getattr(ph, n) for n, _ in ph._fields_])
    want = oracle.o64_deconvolve(v, rph, 0.05, kind=kind, fz2_scale=scale)
    d, out = torch.from_numpy(v).cuda(), torch.empty(shape, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    assert lib.fy_gpu_deconvolve_ex(C.c_void_p(d.data_ptr()), 0, 0.0, 1.0, C.c_void_p(out.data_ptr()), *shape, C.byref(ph),
                                    0.05, kind, scale, None) == 0
    torch.cuda.synchronize()
    assert np.abs(out.cpu().numpy() - want).max() < 16 * max(1.0, math.log2(p)) * 2.0 ** -24
