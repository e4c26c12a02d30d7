"""Phase correlation of several pairs per launch: each pair's result equals the pair's own call bit for
bit (tolerance: none), for axis lengths with a compile-time plan, without one, and mixed; the integer
peak equals the FP64 oracle's."""
import ctypes as C

import numpy as np
import pytest

from tests.test_gpu_phasecorr import gpu_pc, o64_pc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,pairs,window", [((40, 48, 56), 5, 1), ((20, 24, 30), 3, 0), ((33, 70, 130), 2, 1),
                                                ((5, 260, 300), 3, 0), ((6, 7, 600), 2, 0), ((2, 2, 2), 4, 0)])
def test_pairs_at_once(gpu, shape, pairs, window):
    import torch
    lib = gpu.load()
    rng = np.random.default_rng(sum(shape))
    f = rng.uniform(0, 1, (pairs, *shape)).astype(np.float32)
    m = np.stack([np.roll(f[i], (i, -i, 1), (0, 1, 2)) for i in range(pairs)])
    f[-1] = m[-1] = 0.5                                      # flat volumes: degenerate, beside others that are not
    d_f, d_m = torch.from_numpy(f).cuda(), torch.from_numpy(m).cuda()
    scratch = torch.empty(lib.fy_gpu_phase_correlate_scratch_bytes(*shape), dtype=torch.uint8, device="cuda")
    sh, pk = (C.c_double * (3 * pairs))(), (C.c_double * pairs)()
    ix, st = (C.c_longlong * pairs)(), (C.c_int * pairs)()
    torch.cuda.synchronize()
    assert lib.fy_gpu_phase_correlate_batch(C.c_void_p(d_f.data_ptr()), C.c_void_p(d_m.data_ptr()), pairs, *shape, window,
                                            C.c_void_p(scratch.data_ptr()), sh, pk, ix, st, None) == 0
    assert st[pairs - 1] == 1 and sh[3 * pairs - 1] == 0.0
    for i in range(pairs - 1):
        rc, s1, p1 = gpu_pc(gpu, f[i], m[i], window)
        assert rc == 0 == st[i] and list(s1) == list(sh[3 * i:3 * i + 3]) and p1 == pk[i]
        if min(shape) > 2:
            assert ix[i] == o64_pc(f[i], m[i], window)[3]
