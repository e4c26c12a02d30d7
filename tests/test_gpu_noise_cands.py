"""The noise model's radix passes over the windows' candidates: forced, and on a field that sends the means
there by itself. They select the same exact order statistics as the windows (tolerance: none), and
the hook tells that they ran."""
import ctypes as C

import pytest

from tests.test_gpu_noise import gpu_noise
from tests.test_gpu_noise_windows import _volume

pytestmark = pytest.mark.gpu


def _run(gpu, vol, force):
    lib, used = gpu.load(), C.c_int(-1)
    try:
        assert lib.fy_gpu_test_noise_paths(force, None) == 0
        m = gpu_noise(gpu, vol, 5, 10.0, 0.4)
    finally:
        assert lib.fy_gpu_test_noise_paths(0, C.byref(used)) == 0
    return (m.g, m.b, m.noise_ref, m.n_bins_used), used.value


@pytest.mark.parametrize("shape", [(64, 64, 64), (37, 53, 91), (100, 128, 96)])
def test_forced(gpu, shape):
    vol = _volume("smooth", shape)
    want, used = _run(gpu, vol, 0)
    assert used == 3
    for force in (4, 8, 12):
        got, used = _run(gpu, vol, force)
        assert got == want and used == 3 | force


def test_ties(gpu):
    """Four planes of zero means: 49152 equal keys around the 1st percentile, more than a target collects."""
    vol = _volume("masked", (100, 128, 96))
    got, used = _run(gpu, vol, 0)
    assert used & 5 == 5
    assert _run(gpu, vol, 1)[0] == got
