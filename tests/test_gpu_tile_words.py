"""The despeckle's material bits at the words' edges, against the oracle's per-tile chain.

The components are found on 32-voxel words of a row: what can go wrong lies where a run, a
component or the inner tile crosses a word, in rows that end in one, and in a word that is all
material. The chain runs without its float stages, so the bytes and the air state are the oracle's.
"""
import numpy as np
import pytest

import oracle
from tests._tiles import gpu_process_buffer

pytestmark = pytest.mark.gpu


def _volume(nx, kind):
    rng = np.random.default_rng(nx)
    v = np.zeros((9, 12, nx), np.uint8)
    if kind == "noise":                       # many short runs, joined in every direction
        v[rng.random(v.shape) < 0.2] = 180
    elif kind == "solid":                     # words that are all material, and holes in them
        v[2:7, 2:10, 1:-1] = 180
        v[rng.random(v.shape) < 0.3] = 0
    else:                                     # single rows that end or start at a word's edge
        for k, x in enumerate(range(0, nx - 1, 31)):
            v[1 + k % 7, 1 + k % 10, x:x + 2 + 5 * (k % 3)] = 180
            v[1 + (k + 3) % 7, 1 + (k + 5) % 10, max(0, x - 3):x + 1] = 180
    return v


@pytest.mark.parametrize("kind", ["noise", "solid", "edges"])
@pytest.mark.parametrize("nx", [31, 32, 33, 64, 65, 97, 1057])
def test_word_edges(gpu, nx, kind):
    v = _volume(nx, kind)
    d = oracle.pipeline_defaults(air_min_component=12, air_cut_u8=0, air_cut_band=0, air_thresh=1e-9)
    inner = (1, 1, 3, 7, 10, nx - 4)          # three voxels in: the inner rows start inside a word
    rc, g, _ = gpu_process_buffer(gpu, d, v, (0, 0, 0), inner, v.shape[1:])
    assert rc == 0, gpu.load().fy_gpu_last_error()
    o, _ = oracle.ot_process_buffer(d, v, (0, 0, 0), inner, v.shape[1:])
    assert np.array_equal(g, o), np.count_nonzero(g != o)
