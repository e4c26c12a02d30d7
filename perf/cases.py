"""The workloads this library is timed on: calls that programs make, through the public entry points.

Sizes are those of the benchmark's configurations (512^3 cubes with rings, 128^3 cubes, uneven batches
of 96..320 per axis, 256^3 registration pairs, 144^3 export tiles, 8x512x512 viewer slabs) and of the
tests (small and odd shapes). Inputs are seeded phantoms made as the benchmark makes them.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import fysics_b200 as fb
from fysics_b200 import phantom as ph

NB = 24                      # intensity bins of the noise model
LUTN = 4096                  # entries of the deconvolution's radial weight table
BATCH_DIMS = (96, 128, 160, 200, 240, 256, 320)


# ---------------------------------------------------------------------------------- the cases
def listed():
    return [
        # the production cube: dewindow, matched anisotropic deconvolution, noise model, guided
        # filter, ring vote and subtraction (the benchmark's configuration)
        dict(name="restore_512_rings", kind="restore", nz=512, ny=512, nx=512, deconv=1, rings=True),
        # a serving request of the middle class, no rings
        dict(name="restore_256", kind="restore", nz=256, ny=256, nx=256, deconv=1, rings=False),
        # the smallest benchmark cube: isotropic Paganin deconvolution
        dict(name="restore_128", kind="restore", nz=128, ny=128, nx=128, deconv=0, rings=False),
        # a crop at a volume's face, as the tests take them: odd sides, rows of no alignment
        dict(name="restore_61x75x91", kind="restore", nz=61, ny=75, nx=91, deconv=1, rings=True),
        # uneven cubes restored in one call
        dict(name="batch_16_uneven", kind="batch", count=16, lo=96, hi=320),
        # one volume in float through the deconvolution alone, automatic regularisation
        dict(name="deconvolve_256", kind="deconvolve", nz=256, ny=256, nx=256, deconv=0, u8=False),
        # a haloed 128^3 tile of the reference's own timing table, from bytes, matched filter
        dict(name="deconvolve_176_u8", kind="deconvolve", nz=176, ny=176, nx=176, deconv=1, u8=True),
        # the viewer's slab on host memory, one synchronous call
        dict(name="slab_host_8x512x512", kind="slab_host", nz=8, ny=512, nx=512),
        # noise model, then the exact guided filter with its eps, on a ragged volume
        dict(name="denoise_160x208x250", kind="denoise", nz=160, ny=208, nx=250, s=1),
        # registration of volume pairs, one batched call
        dict(name="phasecorr_256x4", kind="phasecorr", nz=256, ny=256, nx=256, pairs=4, window=0),
        # registration of small patches with a Hann window, padded to powers of two
        dict(name="phasecorr_56x72x96x8", kind="phasecorr", nz=56, ny=72, nx=96, pairs=8, window=1),
        # one export tile of 128^3 with its 8-voxel halo, bytes in and out
        dict(name="tile_144", kind="tile", tile=128, halo=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["restore", "restore", "restore", "batch", "deconvolve", "deconvolve", "slab_host", "denoise",
                       "denoise", "phasecorr", "tile"])
    if kind == "restore":
        nz, ny, nx = (_log(rng, 56, 512) for _ in range(3))
        if rng.random() < 0.5:
            nx = min(512, (nx + 3) // 4 * 4)
        return dict(kind=kind, nz=nz, ny=ny, nx=nx, deconv=rng.choice([0, 1]), rings=rng.random() < 0.5)
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(4, 16), lo=rng.choice([96, 128]), hi=rng.choice([200, 256, 320]))
    if kind == "deconvolve":
        nz = rng.choice([8, _log(rng, 24, 400)])
        return dict(kind=kind, nz=nz, ny=_log(rng, 48, 512), nx=_log(rng, 48, 512), deconv=rng.choice([0, 1]),
                    u8=rng.random() < 0.5)
    if kind == "slab_host":
        return dict(kind=kind, nz=rng.randint(4, 16), ny=_log(rng, 192, 768), nx=_log(rng, 192, 768))
    if kind == "denoise":
        nz, ny, nx = (_log(rng, 48, 320) for _ in range(3))
        return dict(kind=kind, nz=nz, ny=ny, nx=nx, s=rng.choice([1, 1, 2]))
    if kind == "phasecorr":
        nz, ny, nx = (_log(rng, 40, 256) for _ in range(3))
        return dict(kind=kind, nz=nz, ny=ny, nx=nx, pairs=rng.randint(1, 6), window=rng.choice([0, 1]))
    return dict(kind=kind, tile=_log(rng, 48, 144), halo=rng.choice([4, 8, 12]))


# ---------------------------------------------------------------------------------- inputs
def _physics(deconv, scale=1.0):
    """The benchmark's physics: config 1 (7.91 um voxels) for the isotropic deconvolution, config 2
    (2.4 um, anisotropic PSF, delta/beta scaled by fy_auto_deltabeta_scale) for the matched one."""
    if deconv == 0:
        return fb.physics(delta_beta=500.0 * scale, energy_kev=110.0, distance_mm=1200.0, pixel_um=7.91,
                          unsharp_sigma=0.8, unsharp_coeff=0.5)
    p = fb.physics(delta_beta=500.0 * scale, energy_kev=110.0, distance_mm=1200.0, pixel_um=2.4, unsharp_sigma=0.8,
                   unsharp_coeff=0.5, psf_sigma_vox=1.0, psf_sigma_z_vox=1.17)
    p.delta_beta *= fb.load().fy_auto_deltabeta_scale(C.byref(p))
    return p


def _phantom(shape, seed, deconv, rings=False, as_float=False):
    p = _physics(deconv)
    return ph.phantom(shape, seed=seed, delta_beta=p.delta_beta, pixel_um=p.pixel_um,
                      fz2_scale=1.17 ** 2 if deconv else 1.0, rings=40 if rings else 0, device="cuda",
                      return_float=as_float)


def _restore_cfg(deconv, ring_handle=None):
    cfg = fb.RestoreCfg()
    fb.load().fy_restore_cfg_default(C.byref(cfg))
    cfg.deconv_kind = deconv
    cfg.deconv_param = 0.05 if deconv == 1 else 0.015
    cfg.dering = ring_handle
    cfg.dering_accumulate = 1 if ring_handle else 0
    return cfg


class _Rings:
    """A device ring state, destroyed with the object."""

    def __init__(self, shape):
        self.lib, self.h = fb.load(), C.c_void_p()
        fb.check(self.lib.fy_gpu_dering_create(C.byref(self.h), *shape, -1.0, -1.0, 512, 8), "fy_gpu_dering_create")

    def __del__(self):
        torch.cuda.synchronize()
        self.lib.fy_gpu_dering_destroy(self.h)


def _batch_shapes(case, seed):
    dims = [d for d in BATCH_DIMS if case["lo"] <= d <= case["hi"]]
    rng = np.random.default_rng(case["count"] * 1000 + case["lo"] + case["hi"])   # the sizes belong to the case
    return [tuple(int(d) for d in rng.choice(dims, 3)) for _ in range(case["count"])]


def _tile_cfg(halo):
    """The export tool's settings: no deconvolution, guided eps on 2x-subsampled coefficients, air cut,
    despeckle of islands under 64 voxels, recenter, dithered bytes."""
    cfg = fb.PipelineCfg()
    for k, v in dict(delta_beta=1000.0, energy_kev=78.0, distance_mm=220.0, pixel_um=2.4, unsharp_sigma=1.2,
                     unsharp_coeff=4.0, use_matched_deconv=1, psf_sigma_vox=1.0, deconv_tikhonov=0.05,
                     guided_eps=8e-4, do_air_zero=1, air_cut_u8=-1, air_cut_band=8, air_thresh=0.05, air_cut_aggr=0.5,
                     air_min_component=64, scratch_passes=5, have_norm=1, norm_lo=40, norm_hi=200, halo=halo,
                     dering_cy=-1.0, dering_cx=-1.0).items():
        setattr(cfg, k, v)
    return cfg


def _pairs(case, seed):
    """Volume pairs: the moving one is an FP64 Fourier shift of the fixed one (integer part up to an
    eighth of the side, and a subvoxel part), each with independent Poisson-Gaussian noise."""
    shape = (case["nz"], case["ny"], case["nx"])
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    f = _phantom(shape, seed, 1, as_float=True).double()
    F = torch.fft.fftn(f)
    k = [torch.fft.fftfreq(n, device="cuda", dtype=torch.float64) for n in shape]
    fixed, moving = [], []
    for _ in range(case["pairs"]):
        s = [int(rng.integers(-n // 8, n // 8 + 1)) + rng.uniform(-0.5, 0.5) for n in shape]
        ang = -2 * math.pi * (k[0][:, None, None] * s[0] + k[1][None, :, None] * s[1] + k[2][None, None, :] * s[2])
        m = torch.fft.ifftn(F * torch.polar(torch.ones_like(ang), ang)).real
        for v, to in ((f, fixed), (m, moving)):
            to.append((v + torch.sqrt(0.002 * v.clamp(min=0) + 1e-4)
                       * torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64)).float())
    return torch.stack(fixed), torch.stack(moving)


def _ptr(t):
    return C.c_void_p(t.data_ptr())


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _shape(case):
    return case["nz"], case["ny"], case["nx"]


def prepare(case, seed):
    lib = fb.load()
    s = dict(case=case, lib=lib)
    kind = case["kind"]
    if kind == "restore":
        shape = _shape(case)
        s["u8"] = _phantom(shape, seed, case["deconv"], case["rings"])
        s["out"] = torch.empty(shape, dtype=torch.float32, device="cuda")
        s["rings"] = _Rings(shape) if case["rings"] else None
        s["phys"] = _physics(case["deconv"])
        s["cfg"] = _restore_cfg(case["deconv"], s["rings"].h.value if case["rings"] else None)
    elif kind == "batch":
        shapes = _batch_shapes(case, seed)
        s["u8"] = [_phantom(sh, seed * 100 + i, 1) for i, sh in enumerate(shapes)]
        s["out"] = [torch.empty(sh, dtype=torch.float32, device="cuda") for sh in shapes]
        s["items"] = (fb.BatchCube * len(shapes))()
        for i, sh in enumerate(shapes):
            it = s["items"][i]
            it.u8, it.out = s["u8"][i].data_ptr(), s["out"][i].data_ptr()
            it.nz, it.ny, it.nx = sh
            it.f32_min, it.f32_max, it.phys = 0.0, 1.0, _physics(1, 0.4 + 0.1 * i)
        s["cfg"] = _restore_cfg(1)
    elif kind == "deconvolve":
        shape = _shape(case)
        s["in"] = _phantom(shape, seed, case["deconv"], as_float=not case["u8"])
        s["out"] = torch.empty(shape, dtype=torch.float32, device="cuda")
        s["phys"] = _physics(case["deconv"])
    elif kind == "slab_host":
        s["in"] = np.random.default_rng(seed).uniform(0.0, 1.0, _shape(case)).astype(np.float32)
        s["phys"] = fb.physics()
    elif kind == "denoise":
        shape = _shape(case)
        s["in"] = _phantom(shape, seed, 1, as_float=True)
        s["out"] = torch.empty(shape, dtype=torch.float32, device="cuda")
        s["scratch"] = torch.empty(lib.fy_gpu_noise_scratch_bytes(*shape), dtype=torch.uint8, device="cuda")
    elif kind == "phasecorr":
        s["fixed"], s["moving"] = _pairs(case, seed)
        s["scratch"] = torch.empty(lib.fy_gpu_phase_correlate_scratch_bytes(*_shape(case)), dtype=torch.uint8,
                                   device="cuda")
    elif kind == "tile":
        h, t = case["halo"], case["tile"]
        side = t + 2 * h
        # the tile sits off the scroll's axis, so that it holds air, body and masked voxels
        vol = ph.scroll_volume((side, 2 * side, 2 * side), seed=seed)
        s["vyx"] = vol.shape[1:]
        s["u8"] = torch.from_numpy(np.ascontiguousarray(vol[:, :side, side // 2:side // 2 + side])).cuda()
        s["org"], s["inner"] = (0, 0, side // 2), (h, h, side // 2 + h, t, t, t)
        s["out"] = torch.empty((t, t, t), dtype=torch.uint8, device="cuda")
        s["cfg"] = _tile_cfg(h)
    return s


# ---------------------------------------------------------------------------------- one pass
def run(s):
    case, lib = s["case"], s["lib"]
    kind = case["kind"]
    if kind == "restore":
        if s["rings"]:
            fb.check(lib.fy_gpu_dering_reset(s["rings"].h, _stream()), "fy_gpu_dering_reset")
        fb.check(lib.fy_gpu_restore_u8(_ptr(s["u8"]), _ptr(s["out"]), *_shape(case), 0.0, 1.0, C.byref(s["phys"]),
                                       C.byref(s["cfg"]), _stream()), "fy_gpu_restore_u8")
        return s["out"]
    if kind == "batch":
        fb.check(lib.fy_gpu_restore_u8_batch(s["items"], len(s["items"]), C.byref(s["cfg"]), _stream()),
                 "fy_gpu_restore_u8_batch")
        return s["out"]
    if kind == "deconvolve":
        fb.check(lib.fy_gpu_deconvolve_ex(_ptr(s["in"]), int(case["u8"]), 0.0, 1.0, _ptr(s["out"]), *_shape(case),
                                          C.byref(s["phys"]), 0.0, case["deconv"], 1.0, _stream()),
                 "fy_gpu_deconvolve_ex")
        return s["out"]
    if kind == "slab_host":
        return fb.deconvolve(s["in"], s["phys"], -1.0)
    if kind == "denoise":
        nm = fb.NoiseModel()
        fb.check(lib.fy_gpu_estimate_noise(_ptr(s["in"]), *_shape(case), 5, 10.0, 0.4, _ptr(s["scratch"]), _stream()),
                 "fy_gpu_estimate_noise")
        fb.check(lib.fy_gpu_noise_model(_ptr(s["scratch"]), *_shape(case), C.byref(nm), _stream()),
                 "fy_gpu_noise_model")
        eps = lib.fy_guided_eps_for_noise(nm.noise_ref)
        fb.check(lib.fy_gpu_guided(_ptr(s["in"]), _ptr(s["out"]), *_shape(case), 2, eps, case["s"], _stream()),
                 "fy_gpu_guided")
        return {"out": s["out"], "g": nm.g, "b": nm.b, "noise_ref": nm.noise_ref, "bins": nm.n_bins_used}
    if kind == "phasecorr":
        n = case["pairs"]
        shift, peak = (C.c_double * (3 * n))(), (C.c_double * n)()
        index, status = (C.c_longlong * n)(), (C.c_int * n)()
        fb.check(lib.fy_gpu_phase_correlate_batch(_ptr(s["fixed"]), _ptr(s["moving"]), n, *_shape(case),
                                                  case["window"], _ptr(s["scratch"]), shift, peak, index, status,
                                                  _stream()), "fy_gpu_phase_correlate_batch")
        return {"shift": np.array(shift), "peak": np.array(peak), "index": np.array(index), "status": np.array(status)}
    if kind == "tile":
        air = C.c_int()
        fb.check(lib.fy_gpu_process_buffer(C.byref(s["cfg"]), _ptr(s["u8"]), *s["org"], *s["u8"].shape, *s["inner"],
                                           *s["vyx"], _ptr(s["out"]), C.byref(air), _stream()),
                 "fy_gpu_process_buffer")
        return {"out": s["out"], "all_air": air.value}
    raise ValueError(kind)


# ---------------------------------------------------------------------------------- what a pass needs
def _fft_flops(n):
    """A real transform pair and the weight over n points."""
    return 2 * 2.5 * n * math.log2(max(2, n)) + 6 * n


def work(case):
    kind = case["kind"]
    if kind == "batch":
        n = sum(math.prod(sh) for sh in _batch_shapes(case, 0))
        return {"bytes": 5.0 * n, "flops": _fft_flops(256 ** 3) / 256 ** 3 * n + 90.0 * n}
    if kind == "tile":
        n, m = (case["tile"] + 2 * case["halo"]) ** 3, case["tile"] ** 3
        return {"bytes": float(n + m), "flops": 60.0 * n}
    n = math.prod(_shape(case))
    if kind == "restore":        # bytes in, floats out; transforms, two box statistics, two box means
        return {"bytes": 5.0 * n, "flops": _fft_flops(n) + 90.0 * n}
    if kind == "deconvolve":
        return {"bytes": (1.0 if case["u8"] else 4.0) * n + 4.0 * n, "flops": _fft_flops(n)}
    if kind == "slab_host":
        return {"bytes": 8.0 * n, "flops": _fft_flops(n)}
    if kind == "denoise":
        return {"bytes": 8.0 * n, "flops": 90.0 * n}
    p = math.prod(1 << (d - 1).bit_length() for d in _shape(case))
    return {"bytes": 8.0 * n * case["pairs"], "flops": case["pairs"] * (3 * 2.5 * p * math.log2(p) + 20.0 * p)}


# ---------------------------------------------------------------------------------- 64-bit values
def _reflect(n, p):
    i = torch.arange(p, device="cuda")
    if n == 1:
        return torch.zeros_like(i)
    i = i % (2 * n)
    return torch.where(i < n, i, 2 * n - 1 - i)


def _pad_len(n):
    p2 = 1 << (n - 1).bit_length() if n > 1 else 1
    m = (n + 2) // 3
    p3 = 3 * (1 << (m - 1).bit_length() if m > 1 else 1)
    return p3 if n <= p3 < p2 else p2


def _x_deconvolve(v, p, deconv, param):
    """Reflect-pad, transform, weight from the 4096-entry table over f^2 (linear between entries), invert."""
    shape = v.shape
    pz, py, px = (_pad_len(n) for n in shape)
    fz2s = 1.0
    if deconv == 1:
        param = param if param > 0 else 0.05
        sxy = p.psf_sigma_vox if p.psf_sigma_vox > 0 else 1.0
        fz2s = (p.psf_sigma_z_vox / sxy) ** 2 if p.psf_sigma_z_vox > 0 else 1.0
    elif param <= 0:
        param = fb.load().fy_auto_reg(C.byref(p), 0.015)
    f2 = [(torch.fft.fftfreq(n, device="cuda", dtype=torch.float64) ** 2) * s for n, s in ((pz, fz2s), (py, 1.0))]
    f2.append(torch.fft.rfftfreq(px, device="cuda", dtype=torch.float64) ** 2)
    umax = sum(float(f.max()) for f in f2)
    us = LUTN / umax
    fr2 = torch.arange(LUTN + 1, device="cuda", dtype=torch.float64) / us
    unsharp = 1.0 + p.unsharp_coeff * (1.0 - torch.exp(-2.0 * math.pi ** 2 * p.unsharp_sigma ** 2 * fr2))
    if deconv == 1:
        sg = p.psf_sigma_vox if p.psf_sigma_vox > 0 else 1.0
        h = torch.exp(-2.0 * math.pi ** 2 * sg * sg * fr2) * unsharp
        lut = h / (h * h + param)
    else:
        lam, dist = 1.23984199e-3 / p.energy_kev, p.distance_mm * 1000.0
        h = (unsharp / (1.0 + p.delta_beta * lam * dist * math.pi * fr2 / p.pixel_um ** 2)).clamp(min=1e-4)
        lut = (h / (h * h + param)).clamp(max=8.0)
    if (pz, py, px) != tuple(shape):
        v = v[_reflect(shape[0], pz)][:, _reflect(shape[1], py)][:, :, _reflect(shape[2], px)]
    spec = torch.fft.rfftn(v)
    del v
    for z in range(pz):                                  # plane by plane: the weight of a plane at a time
        t = (f2[0][z] + f2[1][:, None] + f2[2][None, :]) * us
        ti = t.long().clamp(max=LUTN - 1)
        spec[z] *= lut[ti] + (lut[ti + 1] - lut[ti]) * (t - ti)
    out = torch.fft.irfftn(spec, s=(pz, py, px))
    return out[:shape[0], :shape[1], :shape[2]].contiguous()


def _box_sum(v, r):
    for d in range(3):
        n = v.shape[d]
        out = v.clone()
        for o in range(1, r + 1):
            if o < n:
                out.narrow(d, 0, n - o).add_(v.narrow(d, o, n - o))
                out.narrow(d, o, n - o).add_(v.narrow(d, 0, n - o))
        v = out
    return v


def _box_count(shape, r):
    c = [torch.tensor([min(n - 1, i + r) - max(0, i - r) + 1 for i in range(n)], device="cuda", dtype=torch.float64)
         for n in shape]
    return c[0][:, None, None] * c[1][None, :, None] * c[2][None, None, :]


def _pct(v, pct):
    """percentile between the sorted neighbours"""
    n = v.numel()
    idx = pct / 100.0 * (n - 1)
    k = int(idx)
    v = torch.sort(v.reshape(-1)).values
    return float(v[k]) * (1 - (idx - k)) + float(v[k + 1]) * (idx - k) if k + 1 < n else float(v[k])


def _x_noise(v, win, pct, ref):
    wc = float(win ** 3)
    mean = _box_sum(v, win // 2) / wc
    var = (_box_sum(v * v, win // 2) / wc - mean * mean).clamp(min=0)
    lo, hi = _pct(mean, 1.0), _pct(mean, 99.0)
    hi = hi if hi > lo else lo + 1e-6
    bi, bf, bc = [], [], []
    for b in range(NB):
        b0, b1 = lo + (hi - lo) * b / NB, lo + (hi - lo) * (b + 1) / NB
        inb = var[(mean >= b0) & (mean < b1)]
        if inb.numel() >= 200:
            bi.append(0.5 * (b0 + b1))
            bf.append(_pct(inb, pct))
            bc.append(inb.numel())
    x, y, c = np.array(bi), np.array(bf), np.array(bc, dtype=np.float64)
    g = b = 0.0
    if len(x) >= 3:
        w = np.sqrt(c)
        for _ in range(4):
            sw, swx, swy, swxx, swxy = w.sum(), (w * x).sum(), (w * y).sum(), (w * x * x).sum(), (w * x * y).sum()
            det = sw * swxx - swx * swx
            if abs(det) < 1e-20:
                break
            g, b = (sw * swxy - swx * swy) / det, (swxx * swy - swx * swxy) / det
            res = np.abs(y - (g * x + b))
            w = np.sqrt(c) / (1.0 + (res / (2.0 * (np.median(res) + 1e-9))) ** 2)
    elif len(x):
        b = y.mean()
    else:
        b = _pct(var, pct)
    vr = g * ref + b
    vr = vr if vr >= 0 else max(b, 0.0)
    return g, b, math.sqrt(vr) * 1.15, len(x)


def _x_guided(v, r, eps, s=1):
    full, shape = v, v.shape
    low = [-(-n // s) for n in shape]
    if s > 1 and min(low) >= 2:
        v, r = v[::s, ::s, ::s].contiguous(), max(1, r // s)
    cnt = _box_count(v.shape, r)
    m = _box_sum(v, r) / cnt
    var = (_box_sum(v * v, r) / cnt - m * m).clamp(min=0)
    a = var / (var + eps)
    ab = [_box_sum(q, r) / cnt for q in (a, m * (1.0 - a))]
    del m, var, a, cnt
    if v is not full:                                    # trilinear back to the full grid
        for d in range(3):
            u = torch.arange(shape[d], device="cuda", dtype=torch.float64) / s
            i = u.long().clamp(max=low[d] - 2)
            f = (u - i).clamp(max=1.0).reshape([-1 if q == d else 1 for q in range(3)])
            ab = [q.index_select(d, i) * (1 - f) + q.index_select(d, i + 1) * f for q in ab]
    return ab[0] * full + ab[1]


def _x_rings(u8, out, scale):
    """Accumulate on the 2x grid, sector vote, subtraction (one slab of 512 planes at most)."""
    nz, ny, nx = u8.shape
    cy, cx, ns, hw = (ny - 1) / 2.0, (nx - 1) / 2.0, 8, 7
    nr = int(math.sqrt(cy * cy + cx * cx)) + 2
    gy = torch.arange(0, ny, 2, device="cuda", dtype=torch.float64)[:, None] - cy
    gx = torch.arange(0, nx, 2, device="cuda", dtype=torch.float64)[None, :] - cx
    ri = (torch.sqrt(gy * gy + gx * gx) + 0.5).long()
    q = ((torch.atan2(gy.expand_as(ri), gx.expand_as(ri)) + math.pi) * (ns / (2 * math.pi))).long().clamp(max=ns - 1)
    sub = u8[:, ::2, ::2]
    col_sum, col_cnt = sub.sum(0, dtype=torch.int64), (sub > 0).sum(0, dtype=torch.int64)
    idx = (q * nr + ri)[ri < nr]
    sums = torch.zeros(ns * nr, dtype=torch.int64, device="cuda").index_add_(0, idx, col_sum[ri < nr])
    cnts = torch.zeros(ns * nr, dtype=torch.int64, device="cuda").index_add_(0, idx, col_cnt[ri < nr])
    sums, cnts = sums.reshape(ns, nr).cpu().numpy(), cnts.reshape(ns, nr).cpu().numpy()
    ok = cnts >= 100
    prof = np.where(ok, sums / np.maximum(cnts, 1), 0.0)
    hp = np.zeros((ns, nr))
    for s in range(ns):
        for r in range(nr):                              # in order: a dropped radius is not seen by later ones
            if not ok[s, r]:
                continue
            j = np.arange(max(0, r - hw), min(nr - 1, r + hw) + 1)
            j = j[ok[s, j]]
            if len(j) >= hw:
                hp[s, r] = prof[s, r] - prof[s, j].sum() / len(j)
            else:
                ok[s, r] = False
    ring, found = np.zeros(nr), 0
    for r in range(nr):
        h = hp[ok[:, r], r]
        if len(h) < ns - 2 or ((h > 0).any() and (h < 0).any()):
            continue
        m = float(np.median(h))
        if abs(m) >= 0.5:
            ring[r] = min(6.0, max(-6.0, m))
            found += 1
    if found < 2:
        return out
    gy = torch.arange(ny, device="cuda", dtype=torch.float64)[:, None] - cy
    gx = torch.arange(nx, device="cuda", dtype=torch.float64)[None, :] - cx
    ri = (torch.sqrt(gy * gy + gx * gx) + 0.5).long()
    val = torch.where(ri < nr, torch.from_numpy(ring).cuda()[ri.clamp(max=nr - 1)], torch.zeros_like(gy * gx)) * scale
    return torch.where((out > 0) & (ri < nr), (out - val).clamp(min=0), out)


def _x_restore(u8, p, deconv, rings):
    d = _x_deconvolve(u8.double() / 255.0, p, deconv, 0.05 if deconv == 1 else 0.015)
    noise_ref = _x_noise(d, 5, 10.0, 0.4)[2]
    out = _x_guided(d, 2, max(1e-8, (3.0 * noise_ref) ** 2))
    return _x_rings(u8, out, 1.0 / 255.0) if rings else out


def _x_phasecorr(f, m, window):
    n = f.shape
    p = [1 << (d - 1).bit_length() for d in n]
    f, m = f.double() - f.double().mean(), m.double() - m.double().mean()
    if window:
        w = [0.5 - 0.5 * torch.cos(2 * math.pi * torch.arange(d, device="cuda", dtype=torch.float64) / (d - 1)) for d in n]
        w = w[0][:, None, None] * w[1][None, :, None] * w[2][None, None, :]
        f, m = f * w, m * w
    c = torch.conj(torch.fft.rfftn(f, s=p)) * torch.fft.rfftn(m, s=p)
    mag = c.abs()
    c = torch.where(mag > 1e-12, c / mag.clamp(min=1e-300), torch.zeros_like(c))
    surf = torch.fft.irfftn(c, s=p) * math.prod(p)
    at = int(surf.argmax())
    k = [at // (p[1] * p[2]), at // p[2] % p[1], at % p[2]]
    c0, shift = float(surf[tuple(k)]), []
    for a in range(3):
        lobe = [float(surf[tuple((k[d] + o) % p[d] if d == a else k[d] for d in range(3))]) for o in (-1, 1)]
        c1, sg = (lobe[1], 1.0) if lobe[1] >= lobe[0] else (lobe[0], -1.0)
        d1, d2 = c1 / (c1 - c0), c1 / (c1 + c0)
        d = sg * (d1 if abs(d1) <= abs(d2) else d2)
        shift.append((k[a] if k[a] <= p[a] // 2 else k[a] - p[a]) + min(0.5, max(-0.5, d)))
    return shift, c0 / math.prod(p), at


def exact(case, seed):
    kind = case["kind"]
    if kind == "tile":
        return None                                      # bytes in, bytes out
    s = prepare(case, seed)
    if kind == "restore":
        return _x_restore(s["u8"], s["phys"], case["deconv"], case["rings"])
    if kind == "batch":
        return [_x_restore(u, it.phys, 1, False) for u, it in zip(s["u8"], s["items"])]
    if kind == "deconvolve":
        v = s["in"].double()
        return _x_deconvolve(v / 255.0 if case["u8"] else v, s["phys"], case["deconv"], 0.0)
    if kind == "slab_host":
        return _x_deconvolve(torch.from_numpy(s["in"]).cuda().double(), s["phys"], 0, -1.0).cpu().numpy()
    if kind == "denoise":
        v = s["in"].double()
        g, b, ref, bins = _x_noise(v, 5, 10.0, 0.4)
        return {"out": _x_guided(v, 2, max(1e-8, (3.0 * ref) ** 2), case["s"]), "g": g, "b": b, "noise_ref": ref,
                "bins": bins}
    got = [_x_phasecorr(f, m, case["window"]) for f, m in zip(s["fixed"], s["moving"])]
    return {"shift": np.array([v for g in got for v in g[0]]), "peak": np.array([g[1] for g in got]),
            "index": np.array([g[2] for g in got]), "status": None}
