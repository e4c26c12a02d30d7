"""The noise model's sample-guided windows on the fields that strain their steps: every path selects
the same exact order statistics, so the model equals the radix passes' bit for bit (tolerance: none),
and the FP64 oracle's as tests/test_gpu_noise.py states."""
import ctypes as C

import numpy as np
import pytest

from tests.test_gpu_noise import close, gpu_noise, o64_noise

pytestmark = pytest.mark.gpu


def _volume(kind, shape):
    rng = np.random.default_rng(len(kind) + sum(shape))
    z, y, x = np.meshgrid(*[np.linspace(0, 1, s) for s in shape], indexing="ij")
    v = 0.3 + 0.5 * x * (0.5 + 0.5 * np.sin(3 * y + 2 * z))
    v = (v + rng.standard_normal(shape) * np.sqrt(0.002 * v + 1e-4)).astype(np.float32)
    if kind == "two values":                     # means and variances tie by the thousand
        v = np.where(v > 0.45, np.float32(0.5), np.float32(0.25))
    elif kind == "bytes":                        # a dewindowed u8 volume, never deconvolved
        v = (np.clip(np.rint(v * 255), 0, 255) / 255).astype(np.float32)
    elif kind == "masked":                       # a zero slab: ties of the lowest mean and variance
        v[: shape[0] // 16] = 0
    elif kind == "outliers":                     # a few voxels stretch the sampled range
        v.reshape(-1)[rng.integers(0, v.size, 40)] = 1e6
    elif kind == "not finite":
        v.reshape(-1)[rng.integers(0, v.size, 30)] = np.inf
        v.reshape(-1)[rng.integers(0, v.size, 30)] = -np.inf
        v.reshape(-1)[rng.integers(0, v.size, 30)] = np.nan
    return v


@pytest.mark.parametrize("kind", ["smooth", "two values", "bytes", "masked", "outliers", "not finite"])
@pytest.mark.parametrize("shape", [(64, 64, 64), (37, 53, 91), (100, 128, 96)])
def test_paths_agree(gpu, kind, shape):
    lib, vol = gpu.load(), _volume(kind, shape)
    models = []
    try:
        for force in (0, 1, 2, 3):
            assert lib.fy_gpu_test_noise_paths(force, None) == 0
            g = gpu_noise(gpu, vol, 5, 10.0, 0.4)
            models.append(np.array([g.g, g.b, g.noise_ref, g.n_bins_used]))
    finally:
        lib.fy_gpu_test_noise_paths(0, None)
    for m in models[1:]:
        assert np.array_equal(m, models[0], equal_nan=True), (kind, models)
    if kind in ("smooth", "bytes", "masked"):
        o = o64_noise(vol, 5, 10.0, 0.4)
        assert models[0][3] == o.n_bins_used and close(models[0][2], o.noise_ref)


@pytest.mark.parametrize("n", [1, 5, 63, 64, 65, 199, 200, 217])
def test_few_voxels(gpu, n):
    """No bin, one bin, samples of fewer than 64 values."""
    vol = (0.5 + 0.05 * np.random.default_rng(n).standard_normal((1, 1, n))).astype(np.float32)
    g, o = gpu_noise(gpu, vol, 5, 10.0, 0.4), o64_noise(vol, 5, 10.0, 0.4)
    assert g.n_bins_used == o.n_bins_used and close(g.noise_ref, o.noise_ref)
