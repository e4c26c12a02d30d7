"""Phase correlation of more pairs than run at once (256 MB of workspaces): two full groups and a last
one of a single pair. Each pair's result equals the pair's own call bit for bit (tolerance: none)."""
import ctypes as C

import numpy as np
import pytest

from tests.test_gpu_phasecorr import gpu_pc

pytestmark = pytest.mark.gpu


def test_groups(gpu):
    import torch
    lib, shape = gpu.load(), (66, 70, 72)                # padded to 128^3
    bytes_ = lib.fy_gpu_phase_correlate_scratch_bytes(*shape)
    at_once = (256 << 20) // bytes_
    assert at_once > 2
    pairs = 2 * at_once + 1
    rng = np.random.default_rng(5)
    base = rng.uniform(0, 1, shape).astype(np.float32)
    f = np.stack([base * np.float32(1 + i / 64) for i in range(pairs)])
    m = np.stack([np.roll(f[i], (i % 7 - 3, i % 5 - 2, i % 9 - 4), (0, 1, 2)) for i in range(pairs)])
    f[at_once + 1] = m[at_once + 1] = 0.25               # degenerate, in the second group
    d_f, d_m = torch.from_numpy(f).cuda(), torch.from_numpy(m).cuda()
    scratch = torch.empty(bytes_, dtype=torch.uint8, device="cuda")
    sh, pk = (C.c_double * (3 * pairs))(), (C.c_double * pairs)()
    ix, st = (C.c_longlong * pairs)(), (C.c_int * pairs)()
    torch.cuda.synchronize()
    assert lib.fy_gpu_phase_correlate_batch(C.c_void_p(d_f.data_ptr()), C.c_void_p(d_m.data_ptr()), pairs, *shape, 0,
                                            C.c_void_p(scratch.data_ptr()), sh, pk, ix, st, None) == 0
    for i in range(pairs):
        rc, s1, p1 = gpu_pc(gpu, f[i], m[i], 0)
        assert (rc != 0) == (st[i] != 0) == (i == at_once + 1)
        assert list(s1) == list(sh[3 * i:3 * i + 3]) and p1 == pk[i]
