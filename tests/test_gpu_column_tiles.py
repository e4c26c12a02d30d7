"""The column passes' last columns in shared tiles and in tiles of their own, on both sides of the
rule (64-point columns, 17 of them: shared from 3552 planes in a Y pass, 1776 rows in a Z pass).

Oracle: FP64. Tolerance as for the register plans: a transform of P points rounds at most log2(P)
times per direction (2^-24 each), on values of at most 1 times the gain cap of 8."""
import math

import numpy as np
import pytest

import oracle
from tests.test_gpu_deconv import rphys

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(3552, 64, 32), (3551, 50, 32), (64, 2048, 32), (50, 1500, 32)])
def test_last_columns(gpu, shape):
    lib = gpu.load()
    ph = gpu.physics()
    p = math.prod(lib.fy_next_fft_size(d) for d in shape)
    v = np.random.default_rng(sum(shape)).random(shape, dtype=np.float32)
    want = oracle.o64_deconvolve(v, rphys(ph), 0.015, kind=0)
    assert np.abs(gpu.deconvolve(v, ph, 0.015) - want).max() < 16 * math.log2(p) * 2.0 ** -24
