"""Deconvolution passes with a register plan (axis lengths 64 ... 512), each on every axis in turn.

Sizes: the full length (no padding) and the smallest that pads to it, from f32 and from u8 rows,
with an odd number of rows. Oracle: FP64. Tolerance: a transform of P points rounds at most
log2(P) times per direction (2^-24 each), on values of at most 1 times the gain cap of 8:
8 * 2 * log2(P) * 2^-24 < 3e-5 here."""
import ctypes as C
import math

import numpy as np
import pytest

import oracle
from tests.test_gpu_deconv import rphys

pytestmark = pytest.mark.gpu
LENGTHS = [64, 96, 128, 192, 256, 384, 512]
SMALLEST = dict(zip(LENGTHS, [49, 65, 97, 129, 193, 257, 385]))


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("length", LENGTHS)
def test_register_plan(gpu, length, axis):
    import torch
    lib = gpu.load()
    ph = gpu.physics()
    for n in (length, SMALLEST[length]):
        shape = [[n, 5, 7], [5, n, 19], [3, 5, n]][axis]      # 19 pads to 24: one tile of 13 columns
        p = math.prod(lib.fy_next_fft_size(d) for d in shape)
        tol = 16 * math.log2(p) * 2.0 ** -24
        u8 = np.random.default_rng(n + axis).integers(0, 256, shape, dtype=np.uint8)
        f32 = (u8 / np.float32(255)).astype(np.float32)
        want = oracle.o64_deconvolve(f32, rphys(ph), 0.015, kind=0)
        assert np.abs(gpu.deconvolve(f32, ph, 0.015) - want).max() < tol
        d_in, out = torch.from_numpy(u8).cuda(), torch.empty(shape, dtype=torch.float32, device="cuda")
        assert lib.fy_gpu_deconvolve_ex(C.c_void_p(d_in.data_ptr()), 1, 0.0, 1.0, C.c_void_p(out.data_ptr()), *shape,
                                        C.byref(ph), 0.015, 0, 1.0, None) == 0
        torch.cuda.synchronize()
        assert np.abs(out.cpu().numpy() - want).max() < tol + 2.0 ** -23 * 8
