"""The noise model's whole-field radix passes on a field with more chunks than their CTAs take at once,
against the windows (bit for bit) and on a field whose windows miss, against numpy.

The windows miss where one value fills a percentile: here 0.5, more of the field than a candidate list
holds, between two slabs of noise. The percentiles are exact order statistics of the same
float fields, so the two paths' tolerance is none."""
import numpy as np
import pytest

from tests.test_gpu_noise import close, gpu_noise, o64_noise

pytestmark = pytest.mark.gpu


def _models(gpu, vol, forces):
    lib, out = gpu.load(), []
    try:
        for f in forces:
            assert lib.fy_gpu_test_noise_paths(f, None) == 0
            m = gpu_noise(gpu, vol, 5, 10.0, 0.4)
            out.append((m.g, m.b, m.noise_ref, m.n_bins_used))
    finally:
        lib.fy_gpu_test_noise_paths(0, None)
    return out


# 512 threads x 2 CTAs x 148 SMs of the means' passes take 2.4 million voxels a step, the bins' as many
@pytest.mark.parametrize("shape", [(131, 203, 211), (64, 192, 197)])
def test_large_fields(gpu, shape):
    rng = np.random.default_rng(sum(shape))
    v = 0.3 + 0.4 * np.linspace(0, 1, shape[2], dtype=np.float32) + rng.standard_normal(shape).astype(np.float32) * 0.03
    m = _models(gpu, v, (0, 1, 2, 3))
    assert m[1:] == m[:1] * 3


@pytest.mark.parametrize("shape", [(130, 128, 150)])
def test_windows_miss(gpu, shape):
    rng = np.random.default_rng(7)
    v = (0.3 + 0.4 * rng.random(shape, dtype=np.float32))
    v[: shape[0] * 3 // 4] = 0.9                          # the 99th percentile of the means is a tie
    m = _models(gpu, v, (0, 3))
    assert m[0] == m[1]
    o = o64_noise(v, 5, 10.0, 0.4)
    assert m[0][3] == o.n_bins_used and close(m[0][2], o.noise_ref)
