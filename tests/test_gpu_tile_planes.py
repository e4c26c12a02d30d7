"""The scratch smooth's plane pass and its line passes against the oracle's, bit for bit.

The air cut's histogram and cuts are made of every mean, so they show a wrong one. The lengths are
those where the walk changes: lines shorter than the box, with no step, one step and several steps of
the unrolled middle, and a plane too large for shared memory, which goes line by line.
"""
import numpy as np
import pytest

import oracle
from tests._tiles import gpu_process_buffer, scroll_volume

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("passes", [1, 5, 12])
@pytest.mark.parametrize("shape", [(4, 6, 8), (5, 22, 24), (30, 34, 36), (9, 50, 131), (6, 322, 330)])
def test_scratch_means(gpu, shape, passes):
    v = scroll_volume(shape, seed=5)
    v[0, 0, 0] = 90                           # not all air, whatever the phantom holds
    d = oracle.pipeline_defaults(air_min_component=8, scratch_passes=passes)
    inner = (1, 1, 1, shape[0] - 2, shape[1] - 2, shape[2] - 2)
    rc, g, _ = gpu_process_buffer(gpu, d, v, (0, 0, 0), inner, shape[1:])
    assert rc == 0, gpu.load().fy_gpu_last_error()
    o, _, hist, cuts = oracle.ot_process_buffer(d, v, (0, 0, 0), inner, shape[1:], state=True)
    assert np.array_equal(g, o), np.count_nonzero(g != o)
    gh, gc = np.zeros(256, np.int64), np.zeros(3, np.int32)
    assert gpu.load().fy_process_buffer_air_state(gh.ctypes.data, gc.ctypes.data) == 0
    assert np.array_equal(gh, hist) and np.array_equal(gc, cuts)
