"""Helper threads of a host deconvolution take no CPU time while the GPU has the call."""
import ctypes as C
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_helpers_sleep(gpu):
    """The call's device work waits for a user stream that holds the thread's workspaces for about
    half a second (its clock counted in cycles of at most 2 GHz). The calling thread may spend all of the
    call on a core, and moving 16 MB twice takes milliseconds; helpers that look for work meanwhile
    would add a core each. The bound lies half a core above the calling thread's."""
    import torch
    lib, ph, shape = gpu.load(), gpu.physics(), (16, 512, 512)
    vol = np.random.default_rng(1).uniform(0, 1, shape).astype(np.float32)
    out = np.empty_like(vol)
    small, st = torch.zeros((8, 8, 8), device="cuda"), torch.cuda.Stream()

    def call():
        assert lib.fy_deconvolve(vol.ctypes.data, out.ctypes.data, *shape, C.byref(ph), 0.015) == 0

    call()                                               # workspaces and the ring exist
    torch.cuda.synchronize()
    with torch.cuda.stream(st):
        torch.cuda._sleep(1_000_000_000)
    assert lib.fy_gpu_deconvolve_ex(C.c_void_p(small.data_ptr()), 0, 0.0, 1.0, C.c_void_p(small.data_ptr()), 8, 8, 8,
                                    C.byref(ph), 0.015, 0, 1.0, C.c_void_p(st.cuda_stream)) == 0
    w0, c0 = time.perf_counter(), time.process_time()
    call()
    wall, cpu = time.perf_counter() - w0, time.process_time() - c0
    torch.cuda.synchronize()
    assert wall > 0.2, wall                              # the call did wait
    assert cpu < 1.5 * wall, (cpu, wall)
