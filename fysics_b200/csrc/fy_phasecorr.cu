// fy_phasecorr.cu -- sub-voxel translation by phase correlation (fy_phase_correlate,
// phasecorr.c:38-186) on the half-spectrum engine.
//
//   k_pc_means  double-precision means of the UNWINDOWED inputs (phasecorr.c:66-74):
//               per-thread compensated float sums, per-CTA pairs combined once in double
//   k_pc_x      rows: (f - mean_f)*w | (m - mean_m)*w packed as one complex line per row
//               (w = wz*wy*wx, Hann or ones, phasecorr.c:76-87), zero padding to the next
//               power of two, forward FFT, untangle into the F and M half spectra
//   k_pc_y      forward on both spectra in one launch (rows >= ny are zero)
//   k_pc_z      forward Z of F and M columns (planes >= nz zero), phase-only cross power
//               R = conj(F)M/|conj(F)M| (|.| <= 1e-12 -> 0, phasecorr.c:101-109) with the
//               max magnitude tracked, inverse Z of R
//   k_pc_y      inverse (all padded rows)
//   k_pc_c2r    C2R of every padded row -> correlation surface (real part of the inverse,
//               phasecorr.c:118), only its argmax kept: strictly greater wins, ties go to
//               the first index (phasecorr.c:121-122), via one 64-bit atomicMax
//   k_pc_fit    C2R of the five rows around the peak again, then FP64: fftfreq unwrap and
//               Foroosh subvoxel fit per axis (phasecorr.c:127-182)
//
// The transforms are fy_fft.cuh's with the length as a template argument for 64 ... 512 (N > 0),
// the runtime plan for the rest (N = 0): the same arithmetic, so a shift does not depend on which
// ran. One launch serves `npairs` pairs at once (blockIdx.z), each in a workspace of its own.
// Measured per 256^3 pair, one pair at a time: 548 us with runtime plans, the sum of the means on
// one thread (50 us) and the surface written out (65 us); 339 us now (means 29, x 80, y 51 + 27, z
// 81, c2r 48, fit 8). HBM bounds the means, the L1 data path and latency the transforms.
#include <math.h>
#include <vector>

#include "fy_context.h"
#include "fy_deconv.cuh"

using fy::ctx;
using fy::fail;
using fy::fail_cuda;

// Device-resident results of one correlation.
struct PcCtl {
    double sum_f, sum_m;
    float mean_f, mean_m;
    unsigned int maxmag_bits;            // float bits of the largest |conj(F)M| (>= 0)
    unsigned long long best;             // (orderable value << 32) | (0xffffffff - index)
    double shift[3];
    double peak;
    long long peak_index;
    int status;                          // 0 ok, 1 degenerate (flat input)
};

namespace {

// Threads of a tile and the residency that its registers are budgeted for: 64 a thread, 128 in the Z
// kernel, which holds two columns' points.
template <int N, int E> struct Tile {
    static constexpr int nt = N > 0 ? ct_tile_lines(N) * N / E : KB<E>::nt;
    static constexpr int minb = N > 0 ? 1024 / nt : 1, minb_z = N > 0 ? 512 / nt : 1;
};

// One pair's pointers from the launch's arguments and blockIdx.z.
struct PcArgs {
    const float *fix, *mov;              // the first pair; the next n floats further
    const float *wz, *wy, *wx;           // windows, shared
    char* ws;                            // the first pair's workspace; the next wstride bytes further
    size_t wstride, off_specF, off_specM, off_part, off_ctl;
    long n;
    SpecGeom g;
};
struct Pc {
    const float *fix, *mov;
    float2 *F, *M;
    float4* part;
    PcCtl* ctl;
    FY_D explicit Pc(const PcArgs& a) {
        const size_t p = blockIdx.z;
        fix = a.fix + p * a.n;
        mov = a.mov + p * a.n;
        char* w = a.ws + p * a.wstride;
        F = reinterpret_cast<float2*>(w + a.off_specF);
        M = reinterpret_cast<float2*>(w + a.off_specM);
        part = reinterpret_cast<float4*>(w + a.off_part);
        ctl = reinterpret_cast<PcCtl*>(w + a.off_ctl);
    }
};

FY_D uint32_t fkey(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
FY_D float funkey(uint32_t k) {
    const uint32_t u = (k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k;
    return __uint_as_float(u);
}

// ---------------------------------------------------------------- means
__global__ void __launch_bounds__(256) k_pc_means(const __grid_constant__ PcArgs args) {
    fy_pdl_wait();
    const Pc p(args);
    const float* __restrict__ f = p.fix;
    const float* __restrict__ m = p.mov;
    float sf = 0.f, cf = 0.f, sm = 0.f, cm = 0.f;         // Kahan-compensated per thread
    for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < args.n; i += (long)gridDim.x * blockDim.x) {
        float y = __ldg(f + i) - cf, t = sf + y;
        cf = (t - sf) - y; sf = t;
        y = __ldg(m + i) - cm; t = sm + y;
        cm = (t - sm) - y; sm = t;
    }
    __shared__ double red[2][256];
    red[0][threadIdx.x] = (double)sf - (double)cf;
    red[1][threadIdx.x] = (double)sm - (double)cm;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if (threadIdx.x < w) {
            red[0][threadIdx.x] += red[0][threadIdx.x + w];
            red[1][threadIdx.x] += red[1][threadIdx.x + w];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const double a = red[0][0], b = red[1][0];
        const float ah = (float)a, bh = (float)b;
        p.part[blockIdx.x] = make_float4(ah, (float)(a - ah), bh, (float)(b - bh));
    }
}

// One CTA: the parts' sums (FP64, pairwise) -> means. nparts <= 1024.
__global__ void __launch_bounds__(1024) k_pc_means_final(const __grid_constant__ PcArgs args, int nparts) {
    fy_pdl_wait();
    const Pc p(args);
    const int t = threadIdx.x, lane = t & 31;
    const float4 v = t < nparts ? p.part[t] : make_float4(0.f, 0.f, 0.f, 0.f);
    double sf = (double)v.x + (double)v.y, sm = (double)v.z + (double)v.w;
    __shared__ double rf_[32], rm_[32];
    auto warp_sum = [&](double& x) {
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    };
    warp_sum(sf);
    warp_sum(sm);
    if (lane == 0) { rf_[t >> 5] = sf; rm_[t >> 5] = sm; }
    __syncthreads();
    if (t >= 32) return;
    sf = rf_[lane];
    sm = rm_[lane];
    warp_sum(sf);
    warp_sum(sm);
    if (lane) return;
    PcCtl* ctl = p.ctl;
    ctl->sum_f = sf; ctl->sum_m = sm;
    ctl->mean_f = (float)(sf / args.n);                  // phasecorr.c:74
    ctl->mean_m = (float)(sm / args.n);
    ctl->maxmag_bits = 0;
    ctl->best = 0;
    ctl->status = 0;
}

// ---------------------------------------------------------------- X forward (pair packing)
// W rows per CTA, staged line-major (pitch px + 1, odd: conflict-free for the line-strided accesses).
template <int N, int E, int VEC>
__global__ void __launch_bounds__(Tile<N, E>::nt, Tile<N, E>::minb) k_pc_x(const __grid_constant__ PcArgs args, const __grid_constant__ FftPlan pl,
                                                       const float2* __restrict__ tw, int wlog, FastDiv dchunk, FastDiv dhx) {
    fy_pdl_wait();
    extern __shared__ float4 smem4[];
    const Pc p(args);
    const SpecGeom& g = args.g;
    const int W = 1 << wlog, LPX = g.px + 1;
    float2* s = reinterpret_cast<float2*>(smem4);
    float2* stw = s + W * LPX;
    __shared__ float swzy[16];
    __shared__ long long soff[16];
    const long Q = (long)g.nz * g.ny, q0 = (long)blockIdx.x * W;
    const float mf = p.ctl->mean_f, mm = p.ctl->mean_m;
    load_twiddles(stw, tw, pl.n);
    for (int l = threadIdx.x; l < W; l += blockDim.x) {
        const long q = q0 + l;
        const int qi = q < Q ? (int)q : 0, z = qi / g.ny, y = qi - z * g.ny;
        swzy[l] = args.wz[z] * args.wy[y];
        soff[l] = q < Q ? ((long long)z * g.py + y) * g.hxp : -1;
    }
    __syncthreads();
    const int nch = g.px / VEC;                          // nx and px are multiples of VEC
    for (int it = threadIdx.x; it < W * nch; it += blockDim.x) {
        const int l = dchunk.div(it), x = (it - l * nch) * VEC;
        const long q = q0 + l;
        float a[VEC], b[VEC], w[VEC];
#pragma unroll
        for (int j = 0; j < VEC; ++j) a[j] = b[j] = w[j] = 0.f;
        const bool in = q < Q && x < g.nx;
        if (in) {
            VecLoad<float, VEC>::run(p.fix + q * g.nx + x, a);
            VecLoad<float, VEC>::run(p.mov + q * g.nx + x, b);
#pragma unroll
            for (int j = 0; j < VEC; ++j) w[j] = swzy[l] * args.wx[x + j];
        }
        float2* d = s + l * LPX + x;
#pragma unroll
        for (int j = 0; j < VEC; ++j) d[j] = in ? make_float2((a[j] - mf) * w[j], (b[j] - mm) * w[j]) : make_float2(0.f, 0.f);
    }
    __syncthreads();
    const Lane ln(wlog);
    float2* line = s + ln.l * LPX;
    fft_line<N, E, 1, -1>(line, 1, ln.tl, pl, stw, [&](int i) { return line[i]; }, [&](int i, float2 v) { line[i] = v; });
    __syncthreads();
    for (int idx = threadIdx.x; idx < W * g.hx; idx += blockDim.x) {
        const int l = dhx.div(idx), k = idx - l * g.hx;
        const long long o = soff[l];
        if (o < 0) continue;
        const int mk = k == 0 ? 0 : g.px - k;
        float2 A, B;
        untangle(s[l * LPX + k], s[l * LPX + mk], A, B);
        p.F[o + k] = A;
        p.M[o + k] = B;
    }
}

// ---------------------------------------------------------------- Y
// The columns of `planes` planes of F, then of M when both != 0 (blockIdx.y).
template <int N, int E, int SIGN>
__global__ void __launch_bounds__(Tile<N, E>::nt, Tile<N, E>::minb) k_pc_y(const __grid_constant__ PcArgs args, const __grid_constant__ rf::ColTiles ct,
                                                       const __grid_constant__ FftPlan pl, const float2* __restrict__ tw, int wlog) {
    fy_pdl_wait();
    extern __shared__ float4 smem4[];
    const Pc p(args);
    const SpecGeom& g = args.g;
    const int W = 1 << wlog;
    float2* s = reinterpret_cast<float2*>(smem4);
    float2* stw = s + pl.n * W;
    const Lane ln(wlog);
    const rf::Column c(ct, g.hx, W, ln.l);
    float2* col = (blockIdx.y ? p.M : p.F) + (size_t)c.row * g.py * g.hxp + c.kx;
    const int nin = !c.valid ? 0 : (SIGN < 0 ? g.ny : g.py);
    fft_line_pre<N, E, ct_pitch(N), SIGN>(s + ln.l, W, ln.tl, pl, stw,
                [&](int i) { return i < nin ? col[(size_t)i * g.hxp] : make_float2(0.f, 0.f); },
                [&]() { load_twiddles(stw, tw, pl.n); },
                [&](int i, float2 v) { if (c.valid) col[(size_t)i * g.hxp] = v; });
}

// ---------------------------------------------------------------- Z: cross power
// |conj(F)M| and conj(F)M/|conj(F)M|
FY_D float2 cross_phase(float2 F, float2 M, float& mag) {
    const float cr = F.x * M.x + F.y * M.y;
    const float ci = F.x * M.y - F.y * M.x;
    mag = sqrtf(cr * cr + ci * ci);
    return mag > 1e-12f ? make_float2(cr / mag, ci / mag) : make_float2(0.f, 0.f);
}
// A transform with a compile-time plan whose result stays in registers: point tl + TPL*m at w[m]
// (the last pass, radix R over j = tl + TPL*b, leaves point j + r*N/R at slot b*R + r).
template <int N, int E, int PS, int SIGN, class LD>
FY_D void line_fft_regs(float2 (&w)[E], float2* __restrict__ sline, int tl, const float2* __restrict__ tw, LD ld) {
    constexpr int R = ct_radix(N, ct_npass(N) - 1);
    float2 v[E];
    int c = 0;
    line_fft_ct<N, E, PS, SIGN>(sline, tl, tw, ld, [&](int, float2 x) { v[c++] = x; });
#pragma unroll
    for (int b = 0; b < E / R; ++b)
#pragma unroll
        for (int r = 0; r < R; ++r) w[b + r * (E / R)] = v[b * R + r];
}
template <int N, int E>
__global__ void __launch_bounds__(Tile<N, E>::nt, Tile<N, E>::minb_z)
k_pc_z(const __grid_constant__ PcArgs args, const __grid_constant__ rf::ColTiles ct, const __grid_constant__ FftPlan pl,
       const float2* __restrict__ tw, int wlog) {
    fy_pdl_wait();
    extern __shared__ float4 smem4[];
    const Pc p(args);
    const SpecGeom& g = args.g;
    const int W = 1 << wlog, n = pl.n;
    float2* s = reinterpret_cast<float2*>(smem4);
    float2* stw = s + n * W * (N > 0 ? 1 : 2);
    __shared__ unsigned int s_max;
    const Lane ln(wlog);
    const rf::Column c(ct, g.hx, W, ln.l);
    const size_t zs = (size_t)g.py * g.hxp, coff = (size_t)c.row * g.hxp + c.kx;
    const int nin = c.valid ? g.nz : 0;
    if (threadIdx.x == 0) s_max = 0u;
    load_twiddles(stw, tw, n);
    __syncthreads();
    float lmax = 0.f;
    auto ldF = [&](int i) { return i < nin ? p.F[coff + (size_t)i * zs] : make_float2(0.f, 0.f); };
    auto ldM = [&](int i) { return i < nin ? p.M[coff + (size_t)i * zs] : make_float2(0.f, 0.f); };
    auto stR = [&](int i, float2 v) { if (c.valid) p.F[coff + (size_t)i * zs] = v; };
    if constexpr (N > 0) {
        // both transforms end, and the inverse begins, on the points tl + TPL*m of the thread
        float2 F[E], M[E];
        line_fft_regs<N, E, ct_pitch(N), -1>(F, s + ln.l, ln.tl, stw, ldF);
        line_fft_regs<N, E, ct_pitch(N), -1>(M, s + ln.l, ln.tl, stw, ldM);
#pragma unroll
        for (int m = 0; m < E; ++m) {
            float mag;
            F[m] = cross_phase(F[m], M[m], mag);
            if (mag > lmax) lmax = mag;
        }
        constexpr int R0 = ct_radix(N, 0);
        int k = 0;                                       // loads come in slot order b*R0 + r
        line_fft_ct<N, E, ct_pitch(N), +1>(s + ln.l, ln.tl, stw,
                    [&](int) { const float2 v = F[k / R0 + (k % R0) * (E / R0)]; ++k; return v; }, stR);
    } else {
        float2* sm = s + n * W;
        fft_line<N, E, 0, -1>(s + ln.l, W, ln.tl, pl, stw, ldF, [&](int i, float2 v) { s[i * W + ln.l] = v; });
        __syncthreads();
        fft_line<N, E, 0, -1>(sm + ln.l, W, ln.tl, pl, stw, ldM, [&](int i, float2 v) { sm[i * W + ln.l] = v; });
        __syncthreads();
        for (int z = ln.tl; z < n; z += blockDim.x >> wlog) {
            float mag;
            s[z * W + ln.l] = cross_phase(s[z * W + ln.l], sm[z * W + ln.l], mag);
            if (mag > lmax) lmax = mag;
        }
        __syncthreads();
        fft_line<N, E, 0, +1>(s + ln.l, W, ln.tl, pl, stw, [&](int i) { return s[i * W + ln.l]; }, stR);
    }
    if (c.valid) atomicMax(&s_max, __float_as_uint(lmax));     // non-negative floats order as uints
    __syncthreads();
    if (threadIdx.x == 0) atomicMax(&p.ctl->maxmag_bits, s_max);
}

// ---------------------------------------------------------------- C2R + argmax
// The lines of a tile: line l transforms the spectrum rows at soff[2l], soff[2l+1] (-1: none) and
// leaves their real rows in s[l*(px+1) + x].x and .y.
template <int N, int E>
FY_D void c2r_tile(const float2* __restrict__ spec, const long long* soff, float2* __restrict__ s, float2* __restrict__ stw,
                   const SpecGeom& g, const FftPlan& pl, const float2* __restrict__ tw, int wlog, const FastDiv& dhx) {
    const int W = 1 << wlog, LPX = g.px + 1, hi_max = g.px - g.hx;
    load_twiddles(stw, tw, pl.n);
    constexpr int kU = 4;                                // loads in flight per thread before any is stored
    const int total = W * g.hx, step = blockDim.x;
    for (int base = threadIdx.x; base < total; base += kU * step) {
        float2 A[kU], B[kU];
        int L[kU], K[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const int idx = base + u * step;
            A[u] = B[u] = make_float2(0.f, 0.f);
            L[u] = -1;
            K[u] = 0;
            if (idx < total) {
                const int l = dhx.div(idx), k = idx - l * g.hx;
                const long long oa = soff[2 * l], ob = soff[2 * l + 1];
                L[u] = l;
                K[u] = k;
                if (oa >= 0) A[u] = spec[oa + k];
                if (ob >= 0) B[u] = spec[ob + k];
            }
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            if (L[u] < 0) continue;
            const int l = L[u], k = K[u];
            s[l * LPX + k] = pack_lo(A[u], B[u]);
            if (k >= 1 && k <= hi_max) s[l * LPX + g.px - k] = pack_hi(A[u], B[u]);
        }
    }
    __syncthreads();
    const Lane ln(wlog);
    float2* line = s + ln.l * LPX;
    fft_line<N, E, 1, +1>(line, 1, ln.tl, pl, stw, [&](int i) { return line[i]; }, [&](int i, float2 v) { line[i] = v; });
    __syncthreads();
}
template <int N, int E>
__global__ void __launch_bounds__(Tile<N, E>::nt, Tile<N, E>::minb) k_pc_c2r(const __grid_constant__ PcArgs args, const __grid_constant__ FftPlan pl,
                                                         const float2* __restrict__ tw, int wlog, FastDiv dhx, FastDiv dpx) {
    fy_pdl_wait();
    extern __shared__ float4 smem4[];
    const Pc p(args);
    const SpecGeom& g = args.g;
    const int W = 1 << wlog, LPX = g.px + 1;
    float2* s = reinterpret_cast<float2*>(smem4);
    __shared__ long long soff[2 * 16];
    __shared__ unsigned long long s_best;
    const long Q = (long)g.pz * g.py, q0 = (long)blockIdx.x * 2 * W;      // every padded row
    if (threadIdx.x == 0) s_best = 0;
    for (int i = threadIdx.x; i < 2 * W; i += blockDim.x) soff[i] = q0 + i < Q ? (long long)(q0 + i) * g.hxp : -1;
    __syncthreads();
    c2r_tile<N, E>(p.F, soff, s, s + W * LPX, g, pl, tw, wlog, dhx);
    // a thread meets each row's points in ascending order, so "greater" keeps the first of equals;
    // the two rows are kept apart and meet as (key, index) pairs
    uint32_t ka = 0, kb = 0;
    size_t ia = 0, ib = 0;
    for (int idx = threadIdx.x; idx < W * g.px; idx += blockDim.x) {
        const int l = dpx.div(idx), x = idx - l * g.px;
        const long qa = q0 + 2 * l;
        const float2 v = s[l * LPX + x];
        if (qa < Q) {
            const uint32_t k = fkey(v.x);
            if (k > ka) { ka = k; ia = (size_t)qa * g.px + x; }
        }
        if (qa + 1 < Q) {
            const uint32_t k = fkey(v.y);
            if (k > kb) { kb = k; ib = (size_t)(qa + 1) * g.px + x; }
        }
    }
    const unsigned long long a = ka ? ((unsigned long long)ka << 32) | (0xffffffffull - ia) : 0ull;
    const unsigned long long b = kb ? ((unsigned long long)kb << 32) | (0xffffffffull - ib) : 0ull;
    atomicMax(&s_best, a > b ? a : b);
    __syncthreads();
    if (threadIdx.x == 0) atomicMax(&p.ctl->best, s_best);
}

// ---------------------------------------------------------------- FP64 Foroosh fit
// One CTA: the rows of the peak and of its y and z neighbours again, each with the partner row it
// was transformed with (rows 2m, 2m + 1 share a line), so their values are the surface's.
template <int N, int E>
__global__ void __launch_bounds__(Tile<N, E>::nt) k_pc_fit(const __grid_constant__ PcArgs args, const __grid_constant__ FftPlan pl,
                                                      const float2* __restrict__ tw, int wlog, FastDiv dhx) {
    fy_pdl_wait();
    extern __shared__ float4 smem4[];
    const Pc p(args);
    const SpecGeom& g = args.g;
    PcCtl* ctl = p.ctl;
    const int pz = g.pz, py = g.py, px = g.px, W = 1 << wlog, LPX = px + 1;
    float2* s = reinterpret_cast<float2*>(smem4);
    __shared__ long long soff[2 * 16];
    __shared__ float s_row[5][3];                          // rows (z,y) of the peak, y-1, y+1, z-1, z+1; at x-1, x, x+1
    const double maxmag = (double)__uint_as_float(ctl->maxmag_bits);
    if (maxmag < 1e-20) {                                  // phasecorr.c:111-114
        if (threadIdx.x == 0) {
            ctl->status = 1;
            ctl->shift[0] = ctl->shift[1] = ctl->shift[2] = 0.0;
            ctl->peak = 0.0;
            ctl->peak_index = -1;
        }
        return;
    }
    const unsigned long long b = ctl->best;
    const size_t pk = 0xffffffffull - (b & 0xffffffffull);
    const float best = funkey((uint32_t)(b >> 32));
    const int kz = (int)(pk / ((size_t)py * px)), ky = (int)((pk / px) % py), kx = (int)(pk % px);
    const long Q = (long)pz * py;
    const long row[5] = {(long)kz * py + ky, (long)kz * py + (ky - 1 + py) % py, (long)kz * py + (ky + 1) % py,
                         (long)((kz - 1 + pz) % pz) * py + ky, (long)((kz + 1) % pz) * py + ky};
    // W lines at a time (W < 5 for the longest rows)
    for (int r0 = 0; r0 < 5; r0 += W) {
        __syncthreads();
        for (int i = threadIdx.x; i < 2 * W; i += blockDim.x) {
            const int r = r0 + (i >> 1);
            const long q = r < 5 ? (row[r] & ~1L) + (i & 1) : Q;
            soff[i] = q < Q ? (long long)q * g.hxp : -1;
        }
        __syncthreads();
        c2r_tile<N, E>(p.F, soff, s, s + W * LPX, g, pl, tw, wlog, dhx);
        if (threadIdx.x == 0)
            for (int r = r0; r < 5 && r < r0 + W; ++r)
                for (int d = 0; d < 3; ++d) {
                    const float2 v = s[(r - r0) * LPX + (kx + d - 1 + px) % px];
                    s_row[r][d] = (row[r] & 1) ? v.y : v.x;
                }
    }
    if (threadIdx.x != 0) return;
    const int kk[3] = {kz, ky, kx}, pp[3] = {pz, py, px};
    const double c0 = best;
    for (int a = 0; a < 3; ++a) {
        const double cm = a == 0 ? s_row[3][1] : (a == 1 ? s_row[1][1] : s_row[0][0]);
        const double cp = a == 0 ? s_row[4][1] : (a == 1 ? s_row[2][1] : s_row[0][2]);
        const double c1 = (cp >= cm) ? cp : cm;             // larger side lobe
        const double sg = (cp >= cm) ? 1.0 : -1.0;
        double d = 0.0;
        if (fabs(c1 - c0) > 1e-20 && fabs(c1 + c0) > 1e-20) {
            const double d1 = c1 / (c1 - c0), d2 = c1 / (c1 + c0);
            d = sg * ((fabs(d1) <= fabs(d2)) ? d1 : d2);
        }
        if (d > 0.5) d = 0.5;
        if (d < -0.5) d = -0.5;
        const int iu = (kk[a] <= pp[a] / 2) ? kk[a] : kk[a] - pp[a];   // fftfreq unwrap
        ctl->shift[a] = iu + d;
    }
    ctl->peak = (double)best / (double)((size_t)pz * py * px);   // phasecorr.c:182
    ctl->peak_index = (long long)pk;
}

// 1-D Hann weights (phasecorr.c:38-42), float cosf as the reference; ones when !window.
void hann(std::vector<float>& w, int n, int window) {
    w.assign((size_t)n, 1.0f);
    if (!window) return;
    if (n == 1) { w[0] = 1.0f; return; }
    for (int i = 0; i < n; i++) w[(size_t)i] = 0.5f - 0.5f * cosf(2.0f * (float)M_PI * i / (float)(n - 1));
}

}  // namespace

// Workspace layout for one correlation of (nz,ny,nx) padded to powers of two.
struct PcLayout {
    SpecGeom g;
    size_t off_specF, off_specM, off_win, off_part, off_ctl, total;
};

static PcLayout pc_layout(int nz, int ny, int nx) {
    PcLayout L{};
    SpecGeom& g = L.g;
    g.nz = nz; g.ny = ny; g.nx = nx;
    g.pz = fy_next_pow2(nz); g.py = fy_next_pow2(ny); g.px = fy_next_pow2(nx);
    g.hx = g.px / 2 + 1;
    g.hxp = (g.hx + 15) & ~15;
    size_t o = 0;
    auto take = [&](size_t bytes) { const size_t at = o; o += (bytes + 255) & ~(size_t)255; return at; };
    L.off_specF = take((size_t)g.pz * g.py * g.hxp * sizeof(float2));
    L.off_specM = take((size_t)g.nz * g.py * g.hxp * sizeof(float2));
    L.off_win = take(((size_t)nz + ny + nx) * sizeof(float));
    L.off_part = take(1024 * sizeof(float4));
    L.off_ctl = take(sizeof(PcCtl));
    L.total = o;
    return L;
}

size_t fy_pc_scratch_bytes(int nz, int ny, int nx) { return pc_layout(nz, ny, nx).total; }

// A launch with the compile-time plan of length n where there is one (N > 0), else the runtime
// plan: body(integral_constant<N>, integral_constant<E>).
template <class F>
static cudaError_t pc_with_len(int n, F&& body) {
    switch (n) {
        case 64: return body(std::integral_constant<int, 64>{}, std::integral_constant<int, 16>{});
        case 128: return body(std::integral_constant<int, 128>{}, std::integral_constant<int, 16>{});
        case 256: return body(std::integral_constant<int, 256>{}, std::integral_constant<int, 16>{});
        case 512: return body(std::integral_constant<int, 512>{}, std::integral_constant<int, 16>{});
        default: return fy_with_e(fy_fft_e(n), [&](auto e) { return body(std::integral_constant<int, 0>{}, e); });
    }
}
template <class... K, class... A>
static cudaError_t pc_launch(void (*k)(K...), dim3 grid, int nt, size_t smem, cudaStream_t st, A... a) {
    const cudaError_t e = fy_smem_optin(k, smem);
    return e != cudaSuccess ? e : fy_launch_pdl(k, grid, dim3(nt), smem, st, a...);
}

// Enqueue the correlations of `npairs` pairs (consecutive volumes; pair i in the workspace at
// ws + i*wstride); win holds the wz|wy|wx windows.
static cudaError_t pc_enqueue(const float* fix, const float* mov, const float* win, char* ws, size_t wstride, int npairs,
                              const PcLayout& L, int sms, cudaStream_t st, int& launches) {
    const SpecGeom& g = L.g;
    PcArgs A{};
    A.fix = fix; A.mov = mov;
    A.wz = win; A.wy = A.wz + g.nz; A.wx = A.wy + g.ny;
    A.ws = ws; A.wstride = wstride;
    A.off_specF = L.off_specF; A.off_specM = L.off_specM; A.off_part = L.off_part; A.off_ctl = L.off_ctl;
    A.n = (long)g.nz * g.ny * g.nx;
    A.g = g;
    const unsigned np = (unsigned)npairs;
    cudaError_t e;
    int nparts = (int)((A.n + 255) / 256);
    if (nparts > 4 * sms) nparts = 4 * sms;
    if (nparts > 1024) nparts = 1024;
    const FftPlan plx = fy_make_plan(g.px), ply = fy_make_plan(g.py), plz = fy_make_plan(g.pz);
    const float2 *twx = fy::twiddles(g.px), *twy = fy::twiddles(g.py), *twz = fy::twiddles(g.pz);
    if (!twx || !twy || !twz) return cudaErrorMemoryAllocation;
    if ((e = pc_launch(k_pc_means, dim3(nparts, 1, np), 256, 0, st, A)) != cudaSuccess) return e;
    if ((e = pc_launch(k_pc_means_final, dim3(1, 1, np), 1024, 0, st, A, nparts)) != cudaSuccess) return e;
    const TileShape tx = fy_tile_shape(g.px), ty = fy_tile_shape(g.py), tz = fy_tile_shape(g.pz);
    const size_t smem_x = ((size_t)tx.W * (g.px + 1) + g.px) * sizeof(float2);
    const size_t smem_y = (size_t)g.py * (ty.W + 1) * sizeof(float2);
    const FastDiv dhx(g.hx), dpx(g.px);
    {   // X forward of the packed pair, four columns at a time where rows are 16-byte aligned
        const bool vec = g.nx % 4 == 0 && g.px % 4 == 0 && ((uintptr_t)fix % 16) == 0 && ((uintptr_t)mov % 16) == 0;
        const dim3 grid((unsigned)(((long)g.nz * g.ny + tx.W - 1) / tx.W), 1, np);
        const FastDiv dch(vec ? g.px / 4 : g.px);
        e = pc_with_len(g.px, [&](auto nc, auto ec) -> cudaError_t {
            constexpr int N = decltype(nc)::value, E = decltype(ec)::value;
            if (vec) return pc_launch(k_pc_x<N, E, 4>, grid, tx.NT, smem_x, st, A, plx, twx, tx.wlog, dch, dhx);
            return pc_launch(k_pc_x<N, E, 1>, grid, tx.NT, smem_x, st, A, plx, twx, tx.wlog, dch, dhx);
        });
        if (e != cudaSuccess) return e;
    }
    // Y pass: forward on both spectra's nz planes, inverse on the pz planes of R
    auto ypass = [&](int planes, bool fwd) -> cudaError_t {
        const rf::ColTiles ct = rf::col_tiles(g.hx, planes, ty.W);
        const dim3 grid(ct.total, fwd ? 2 : 1, np);
        return pc_with_len(g.py, [&](auto nc, auto ec) -> cudaError_t {
            constexpr int N = decltype(nc)::value, E = decltype(ec)::value;
            if (fwd) return pc_launch(k_pc_y<N, E, -1>, grid, ty.NT, smem_y, st, A, ct, ply, twy, ty.wlog);
            return pc_launch(k_pc_y<N, E, +1>, grid, ty.NT, smem_y, st, A, ct, ply, twy, ty.wlog);
        });
    };
    if ((e = ypass(g.nz, true)) != cudaSuccess) return e;
    {   // Z: cross power
        const rf::ColTiles ct = rf::col_tiles(g.hx, g.py, tz.W);
        e = pc_with_len(g.pz, [&](auto nc, auto ec) -> cudaError_t {
            constexpr int N = decltype(nc)::value, E = decltype(ec)::value;
            const size_t smem = (size_t)g.pz * ((N > 0 ? 1 : 2) * tz.W + 1) * sizeof(float2);
            return pc_launch(k_pc_z<N, E>, dim3(ct.total, 1, np), tz.NT, smem, st, A, ct, plz, twz, tz.wlog);
        });
        if (e != cudaSuccess) return e;
    }
    if ((e = ypass(g.pz, false)) != cudaSuccess) return e;
    e = pc_with_len(g.px, [&](auto nc, auto ec) -> cudaError_t {     // C2R + argmax over every padded row, then the fit
        constexpr int N = decltype(nc)::value, E = decltype(ec)::value;
        const dim3 grid((unsigned)(((long)g.pz * g.py + 2 * tx.W - 1) / (2 * tx.W)), 1, np);
        const cudaError_t e2 = pc_launch(k_pc_c2r<N, E>, grid, tx.NT, smem_x, st, A, plx, twx, tx.wlog, dhx, dpx);
        if (e2 != cudaSuccess) return e2;
        return pc_launch(k_pc_fit<N, E>, dim3(1, 1, np), tx.NT, smem_x, st, A, plx, twx, tx.wlog, dhx);
    });
    if (e != cudaSuccess) return e;
    launches += 8;
    return cudaGetLastError();
}

static int pc_check(int nz, int ny, int nx, const char* what) {
    const int pz = fy_next_pow2(nz), py = fy_next_pow2(ny), px = fy_next_pow2(nx);
    if (!fy_fft_len_ok(pz) || !fy_fft_len_ok(py) || !fy_fft_len_ok(px))
        return fail(FY_EUNSUPPORTED, "%s: padded size %dx%dx%d exceeds %d per axis", what, pz, py, px, FY_FFT_MAXN);
    if ((size_t)pz * py * px >= 0xffffffffull)
        return fail(FY_EUNSUPPORTED, "%s: padded volume exceeds 2^32 voxels", what);
    return FY_OK;
}

static int pc_upload_windows(char* ws, const PcLayout& L, int window, cudaStream_t st, std::vector<float>& h) {
    std::vector<float> wz, wy, wx;
    hann(wz, L.g.nz, window); hann(wy, L.g.ny, window); hann(wx, L.g.nx, window);
    h.clear();
    h.insert(h.end(), wz.begin(), wz.end());
    h.insert(h.end(), wy.begin(), wy.end());
    h.insert(h.end(), wx.begin(), wx.end());
    cudaError_t e = cudaMemcpyAsync(ws + L.off_win, h.data(), h.size() * sizeof(float), cudaMemcpyHostToDevice, st);
    return e == cudaSuccess ? FY_OK : fail_cuda(e, "phase correlation windows");
}

extern "C" int fy_phase_correlate(const float* fixed, const float* moving, int nz, int ny, int nx, double* shift,
                                  double* peak, int window) {
    fy::enter();
    const char* what = "fy_phase_correlate";
    if (!fixed || !moving || !shift || nz < 2 || ny < 2 || nx < 2) return 1;   // phasecorr.c:47
    int rc = pc_check(nz, ny, nx, what);
    if (rc) return rc;
    if ((rc = fy::ensure_ctx())) return rc;
    fy::ThreadCtx& c = ctx();
    cudaStream_t st = c.st;
    const PcLayout L = pc_layout(nz, ny, nx);
    const size_t n = (size_t)nz * ny * nx;
    fy::ws_acquire(st);
    cudaError_t e;
    if ((e = c.vin.ensure(2 * n * sizeof(float))) != cudaSuccess) return fail_cuda(e, what);
    if ((e = c.spec.ensure(L.total)) != cudaSuccess) return fail_cuda(e, what);
    if ((e = c.pin.ensure(sizeof(PcCtl))) != cudaSuccess) return fail_cuda(e, what);
    float* dfix = c.vin.as<float>();
    float* dmov = dfix + n;
    char* ws = (char*)c.spec.p;
    std::vector<float> hwin;
    if ((rc = pc_upload_windows(ws, L, window, st, hwin))) return rc;
    if ((e = cudaMemcpyAsync(dfix, fixed, n * 4, cudaMemcpyHostToDevice, st)) != cudaSuccess) return fail_cuda(e, what);
    if ((e = cudaMemcpyAsync(dmov, moving, n * 4, cudaMemcpyHostToDevice, st)) != cudaSuccess) return fail_cuda(e, what);
    int launches = 0;
    if ((e = pc_enqueue(dfix, dmov, (const float*)(ws + L.off_win), ws, L.total, 1, L, c.sms, st, launches)) != cudaSuccess)
        return fail_cuda(e, what);
    fy::count_launch(launches);
    if ((e = cudaMemcpyAsync(c.pin.p, ws + L.off_ctl, sizeof(PcCtl), cudaMemcpyDeviceToHost, st)) != cudaSuccess)
        return fail_cuda(e, what);
    fy::ws_release(st);
    if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return fail_cuda(e, what);
    const PcCtl* r = (const PcCtl*)c.pin.p;
    if (r->status) {
        shift[0] = shift[1] = shift[2] = 0.0;
        if (peak) *peak = 0.0;
        return 1;
    }
    shift[0] = r->shift[0]; shift[1] = r->shift[1]; shift[2] = r->shift[2];
    if (peak) *peak = r->peak;
    return 0;
}

// Device form for batches: `npairs` pairs of device volumes (fixed[i], moving[i] at stride
// nz*ny*nx floats), results written to the host arrays shift[3*npairs], peak[npairs],
// peak_index[npairs] (nullable) and status[npairs]. Synchronises `stream` at the end.
extern "C" size_t fy_gpu_phase_correlate_scratch_bytes(int nz, int ny, int nx) { return fy_pc_scratch_bytes(nz, ny, nx); }

extern "C" int fy_gpu_phase_correlate_batch(const float* d_fixed, const float* d_moving, int npairs, int nz, int ny,
                                            int nx, int window, void* d_scratch, double* shift, double* peak,
                                            long long* peak_index, int* status, void* stream) {
    fy::enter();
    const char* what = "fy_gpu_phase_correlate_batch";
    if (!d_fixed || !d_moving || !d_scratch || !shift || !status || npairs < 0) return fail(FY_EINVAL, "%s: bad args", what);
    if (nz < 2 || ny < 2 || nx < 2) return fail(FY_EINVAL, "%s: dims < 2", what);
    int rc = pc_check(nz, ny, nx, what);
    if (rc) return rc;
    if ((rc = fy::ensure_ctx())) return rc;
    fy::ThreadCtx& c = ctx();
    cudaStream_t st = (cudaStream_t)stream;
    const PcLayout L = pc_layout(nz, ny, nx);
    const size_t n = (size_t)nz * ny * nx;
    char* ws = (char*)d_scratch;
    std::vector<float> hwin;
    if ((rc = pc_upload_windows(ws, L, window, st, hwin))) return rc;
    cudaError_t e;
    if ((e = c.pin.ensure(sizeof(PcCtl) * (size_t)(npairs > 0 ? npairs : 1))) != cudaSuccess) return fail_cuda(e, what);
    PcCtl* host = (PcCtl*)c.pin.p;
    // Small pairs do not fill the GPU one at a time: as many as fit kPairsBytes run in one set of
    // launches, in the thread's workspace (8 pairs of 56x72x96 with a window: 984 us one by one with
    // the former kernels, 160 us together). A pair of 256^3 takes 136 MB and fills the GPU alone.
    constexpr size_t kPairsBytes = (size_t)256 << 20;
    int at_once = (int)(kPairsBytes / L.total < (size_t)npairs ? kPairsBytes / L.total : (size_t)npairs);
    char* pws = ws;
    if (at_once > 1) {
        fy::ws_acquire(st);
        if (c.spec.ensure((size_t)at_once * L.total) == cudaSuccess) pws = (char*)c.spec.p;
        else at_once = 1;                                // no memory for it: one by one in d_scratch
    } else {
        at_once = 1;
    }
    // on every way out, errors among them: launches that use the workspace may be in flight
    struct Release {
        cudaStream_t st;
        bool on;
        ~Release() { if (on) fy::ws_release(st); }
    } release{st, pws != ws};
    int launches = 0;
    for (int i = 0; i < npairs; i += at_once) {
        const int k = npairs - i < at_once ? npairs - i : at_once;
        if ((e = pc_enqueue(d_fixed + (size_t)i * n, d_moving + (size_t)i * n, (const float*)(ws + L.off_win), pws, L.total, k, L,
                            c.sms, st, launches)) != cudaSuccess)
            return fail_cuda(e, what);
        if ((e = cudaMemcpy2DAsync(host + i, sizeof(PcCtl), pws + L.off_ctl, L.total, sizeof(PcCtl), k, cudaMemcpyDeviceToHost,
                                   st)) != cudaSuccess)
            return fail_cuda(e, what);
    }
    fy::count_launch(launches);
    if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return fail_cuda(e, what);
    for (int i = 0; i < npairs; ++i) {
        for (int a = 0; a < 3; ++a) shift[3 * i + a] = host[i].status ? 0.0 : host[i].shift[a];
        if (peak) peak[i] = host[i].status ? 0.0 : host[i].peak;
        if (peak_index) peak_index[i] = host[i].peak_index;
        status[i] = host[i].status;
    }
    return FY_OK;
}
