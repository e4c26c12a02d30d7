// fy_tile.cu -- the export tool's per-tile chain (fy_process_buffer, pipeline.c:252-510) on
// the GPU: one haloed u8 tile in, the inner tile as u8 out.
//
//   k_tile_any      all-air test (pipeline.c:472-476): an empty buffer skips the chain
//   k_tile_prep     u8/255 (pipeline.c:46-48), ring subtraction at scale 1/255
//                   (dering.c:200-248), z drift (zdrift.c:64-71); writes orig and the working
//                   field, windowed to physical units when the deconvolution runs (:271-272)
//   deconvolution   fy_gpu_deconvolve_ex in place: plain auto-reg, or matched (:273-275)
//   k_tile_unwin    re-window, dec-range rescale, clamp to [0, 1] (:277-288)
//   guided filter   fy_gpu_guided, r = 2, subsampled coefficients by default (:290-297)
//   air zero        k_box_plane and k_box_line_smem over the 2x-decimated orig (the sliding sums of
//                   guided.c:34-98; the last pass also bins the means), k_air_cut (stream.c:138-168 and
//                   pipeline.c:330-364), k_air_apply (the texture split, :355-399), which
//                   also writes the despeckle's material bits and x-run heads
//   despeckle       union-find over 6-connected material (:223-250, :400-405): k_cc_union,
//                   k_cc_count (roots, sizes, face contact); the zeroing of small interior
//                   components is applied by the quantiser
//   k_tile_quant    recenter (:407-421) and the dithered quantiser (:53-65, :501-506) over
//                   the inner tile
//
// Arithmetic follows the reference source operation for operation, with its a*b+c forms
// fused and its divisions by constants taken as multiplications by the rounded reciprocal,
// as its build (-Ofast, FMA target) compiles them. The box smooth's 1/count is IEEE: the
// reference build's vectorised reciprocals depend on the host CPU in their last bit. With
// the deconvolution and guided filter off, the output equals the oracle restatement bit for
// bit.
#include "fy_context.h"

#include <math.h>
#include <stdlib.h>
#include <string.h>
#include <algorithm>

using fy::ctx;
using fy::fail;
using fy::fail_cuda;

extern "C" int fy_gpu_deconvolve_ex(const void* d_in, int src_u8, double f32_min, double f32_max, float* d_out,
                                    int nz, int ny, int nx, const fy_physics* p, double param, int kind,
                                    double fz2_scale, void* stream);
extern "C" int fy_gpu_guided(const float* d_in, float* d_out, int nz, int ny, int nx, int radius, double eps, int s,
                             void* stream);

namespace {

constexpr int kUfMaxIter = 1 << 22;      // bound on every union-find walk (never reached in practice)
constexpr unsigned kEdge = 0x80000000u;  // component touches a face of the buffer
constexpr int kTpb = 128;

struct TileCtl {
    int any;                  // the buffer has a nonzero voxel
    int err;                  // a union-find walk hit kUfMaxIter
    unsigned hist[256];       // scratch-smooth histogram
    int cuts[3];              // value cut, uniform cut, textured cut (u8 levels)
    float cutf_uni, cutf_tex;
};

// stream.c:138-168
__host__ __device__ double valley_depth_hd(const long* hist, int* dark_out, int* light_out, int* valley_out) {
    double hf[256];
    for (int i = 0; i < 256; i++) {
        long s = 0;
        int cnt = 0;
        for (int j = i - 2; j <= i + 2; j++)
            if (j >= 0 && j < 256) { s += hist[j]; cnt++; }
        hf[i] = (double)s / cnt;
    }
    hf[0] = 0; hf[254] = 0; hf[255] = 0;
    double mx = 0;
    for (int i = 0; i < 256; i++) mx = hf[i] > mx ? hf[i] : mx;
    if (mx <= 0) return -1;
    int pk[256], np = 0;
    for (int u = 3; u < 253; u++) {
        if (!(hf[u] >= hf[u - 1] && hf[u] >= hf[u + 1] && hf[u] > 0.05 * mx)) continue;
        if (np > 0 && u - pk[np - 1] <= 10) {
            if (hf[u] > hf[pk[np - 1]]) pk[np - 1] = u;
        } else {
            pk[np++] = u;
        }
    }
    if (np < 2) return -1;
    int p1 = pk[0], p2 = pk[1];
    for (int i = 0; i < np; i++) {
        const int u = pk[i];
        if (hf[u] > hf[p1]) { p2 = p1; p1 = u; }
        else if (hf[u] > hf[p2] && u != p1) p2 = u;
    }
    const int a = p1 < p2 ? p1 : p2, b = p1 < p2 ? p2 : p1;
    int v = a;
    double vmin = hf[a];
    for (int u = a; u <= b; u++)
        if (hf[u] < vmin) { vmin = hf[u]; v = u; }
    if (dark_out) *dark_out = a;
    if (light_out) *light_out = b;
    if (valley_out) *valley_out = v;
    const double mn = hf[a] < hf[b] ? hf[a] : hf[b];
    return 1.0 - vmin / (mn + 1e-12);
}

// pipeline.c:53-58
__device__ __forceinline__ float dither01(long z, long y, long x) {
    unsigned h = (unsigned)z * 73856093u ^ (unsigned)y * 19349663u ^ (unsigned)x * 83492791u;
    h ^= h >> 16;
    h *= 0x7feb352du;
    h ^= h >> 15;
    h *= 0x846ca68bu;
    h ^= h >> 16;
    return __fmul_rn((float)(h >> 8), 1.0f / 16777216.0f);
}

// ---------------------------------------------------------------- all-air test
__global__ void __launch_bounds__(256) k_tile_any(const uint8_t* __restrict__ u8, size_t n, TileCtl* ctl) {
    const size_t mis = (size_t)((16 - ((uintptr_t)u8 & 15)) & 15);
    const size_t head = mis < n ? mis : n;
    const size_t nw = (n - head) / 16, tail = head + nw * 16;
    const uint4* w = reinterpret_cast<const uint4*>(u8 + head);
    const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x, nth = (size_t)gridDim.x * blockDim.x;
    unsigned found = 0;
    for (size_t i = tid; i < nw; i += nth) {
        const uint4 v = __ldg(w + i);
        found |= v.x | v.y | v.z | v.w;
    }
    for (size_t i = tid; i < head; i += nth) found |= u8[i];
    for (size_t i = tail + tid; i < n; i += nth) found |= u8[i];
    if (__syncthreads_or(found != 0) && threadIdx.x == 0) ctl->any = 1;
}

// ---------------------------------------------------------------- prep
struct PrepArgs {
    const uint8_t* u8;
    float* orig;
    float* work;              // the deconvolution's input (windowed), or nullptr
    long hz, hy, hx;
    // rings: rows [s0, s0 + rows) of the [nslab][nr] table, or ring == nullptr
    const float* ring;
    long s0, nslab, slab_z;
    int nr;
    double cy, cx;
    long rz0, ry0, rx0;
    float sc;
    const float* zdrift;      // hz factors from global z = rz0, or nullptr
    int windowed;
    float wlo, wspan;
};

// Four consecutive voxels per thread (one 4-byte load, 16-byte stores when aligned).
// Coordinates are derived only when rings or z drift need them.
__device__ __forceinline__ float prep_one(const PrepArgs& a, unsigned u, size_t i, unsigned plane) {
    float f = __fmul_rn((float)u, 1.0f / 255.0f);
    if (a.ring || a.zdrift) {
        const unsigned ii = (unsigned)i;            // hz*hy*hx < 2^31
        const unsigned z = ii / plane, rem = ii - z * plane;
        if (a.ring && f > 0.0f) {
            const unsigned y = rem / (unsigned)a.hx, x = rem - y * (unsigned)a.hx;
            const double gy = (double)(a.ry0 + y) - a.cy, gx = (double)(a.rx0 + x) - a.cx;
            const int r = (int)(sqrt(gy * gy + gx * gx) + 0.5);
            if (r < a.nr) {
                long s = (a.rz0 + (long)z) / a.slab_z;
                s = s < 0 ? 0 : (s >= a.nslab ? a.nslab - 1 : s);
                const float w = __fmaf_rn(-a.sc, __ldg(a.ring + (size_t)(s - a.s0) * a.nr + r), f);
                f = w > 0.0f ? w : 0.0f;
            }
        }
        if (a.zdrift) f = __fmul_rn(f, __ldg(a.zdrift + z));
    }
    return f;
}

__global__ void __launch_bounds__(256) k_tile_prep(PrepArgs a) {
    const size_t n = (size_t)a.hz * a.hy * a.hx;
    const unsigned plane = (unsigned)(a.hy * a.hx);
    const bool vec = ((uintptr_t)a.u8 & 3) == 0;
    for (size_t q = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 4; q < n;
         q += (size_t)gridDim.x * blockDim.x * 4) {
        unsigned u[4] = {0, 0, 0, 0};
        if (vec && q + 4 <= n) {
            const uchar4 v = *reinterpret_cast<const uchar4*>(a.u8 + q);
            u[0] = v.x; u[1] = v.y; u[2] = v.z; u[3] = v.w;
        } else {
            for (int k = 0; k < 4 && q + k < n; k++) u[k] = a.u8[q + k];
        }
        float f[4], w[4];
        for (int k = 0; k < 4; k++) {
            f[k] = prep_one(a, u[k], q + k, plane);
            w[k] = a.windowed ? __fmaf_rn(f[k], a.wspan, a.wlo) : f[k];
        }
        if (q + 4 <= n) {                           // orig and work are 256-byte aligned, q % 4 == 0
            *reinterpret_cast<float4*>(a.orig + q) = make_float4(f[0], f[1], f[2], f[3]);
            if (a.work) *reinterpret_cast<float4*>(a.work + q) = make_float4(w[0], w[1], w[2], w[3]);
        } else {
            for (int k = 0; q + k < n; k++) {
                a.orig[q + k] = f[k];
                if (a.work) a.work[q + k] = w[k];
            }
        }
    }
}

// ---------------------------------------------------------------- after the deconvolution
__global__ void __launch_bounds__(256) k_tile_unwin(float* __restrict__ f, size_t n, int windowed, float wlo,
                                                    float inv, int rescale, float lo, float dinv) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        float v = f[i];
        if (windowed) v = __fmul_rn(__fsub_rn(v, wlo), inv);
        if (rescale) v = __fmul_rn(__fsub_rn(v, lo), dinv);
        f[i] = v < 0.0f ? 0.0f : (v > 1.0f ? 1.0f : v);
    }
}

// ---------------------------------------------------------------- scratch smooth
// One thread per line: prime the sum with samples [0, r], then per sample emit sum/count and
// slide (add the entering sample, then subtract the leaving one), as guided.c:56-95.
struct LineArgs {
    const float* in;
    float* out;
    int L, r;
    long A, B;                // lines = A x B
    long ia, ib, il;          // input strides: outer, inner, along the line
    long oa, ob, ol;
    unsigned* hist;           // staged kernel only: histogram of the means (the air cut's bins)
};

__global__ void __launch_bounds__(kTpb) k_box_line(LineArgs a) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= a.A * a.B) return;
    const long ai = t / a.B, bi = t - ai * a.B;
    const float* in = a.in + ai * a.ia + bi * a.ib;
    float* out = a.out + ai * a.oa + bi * a.ob;
    float s = 0.0f;
    for (int i = 0; i <= a.r && i < a.L; ++i) s = __fadd_rn(s, in[i * a.il]);
    for (int i = 0; i < a.L; ++i) {
        const int lo = i - a.r < 0 ? 0 : i - a.r, hi = i + a.r > a.L - 1 ? a.L - 1 : i + a.r;
        out[i * a.ol] = __fmul_rn(s, __frcp_rn((float)(hi - lo + 1)));
        if (i + a.r + 1 < a.L) s = __fadd_rn(s, in[(i + a.r + 1) * a.il]);
        if (i - a.r >= 0) s = __fsub_rn(s, in[(i - a.r) * a.il]);
    }
}

// The same sliding sums over one line in shared memory. Away from the ends the count is 2r + 1 and
// every step adds one sample and takes one out, so that the loads of several steps go ahead of their
// sums; only the sums themselves are a chain.
__device__ __forceinline__ void line_means(const float* in, float* out, int L, int r, int step) {
    const float rin = __frcp_rn((float)(2 * r + 1));
    float s = 0.0f;
    for (int i = 0; i <= r && i < L; ++i) s = __fadd_rn(s, in[i * step]);
    auto at = [&](int i) {
        const int lo = i - r < 0 ? 0 : i - r, hi = i + r > L - 1 ? L - 1 : i + r;
        out[i * step] = __fmul_rn(s, hi - lo == 2 * r ? rin : __frcp_rn((float)(hi - lo + 1)));
        if (i + r + 1 < L) s = __fadd_rn(s, in[(i + r + 1) * step]);
        if (i - r >= 0) s = __fsub_rn(s, in[(i - r) * step]);
    };
    int i = 0;
    for (; i < r && i < L; ++i) at(i);
    for (; i + r + 1 + 8 <= L; i += 8) {
        float enter[8], leave[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            enter[k] = in[(i + k + r + 1) * step];
            leave[k] = in[(i + k - r) * step];
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            out[(i + k) * step] = __fmul_rn(s, rin);
            s = __fsub_rn(__fadd_rn(s, enter[k]), leave[k]);
        }
    }
    for (; i < L; ++i) at(i);
}

// The x and the y pass in one: a CTA holds a whole (decimated) plane in shared memory, a thread per
// row and then one per column, pitch odd so that both walks are free of bank conflicts. The plane is
// read once and written once, and one launch is saved. Taken where two copies of the plane fit
// (to about 158 x 158 decimated, a buffer of 316 x 316); planes above that go line by line. Measured at
// 144^3 (72 planes of 72 x 72): 18.0 us against 17.7 + 10.5; the z pass, with line_means, 9.3 against 11.3.
struct PlaneArgs {
    const float* in;
    float* out;
    int ny, nx, r;
    long iz, iy, ix;          // input strides; the output is dense
};
constexpr int kPlaneThreads = 256;
__global__ void __launch_bounds__(kPlaneThreads) k_box_plane(PlaneArgs a) {
    extern __shared__ float sl[];
    const int p = a.nx | 1, n = a.ny * a.nx;
    float* so = sl + (size_t)a.ny * p;
    const float* in = a.in + (long)blockIdx.x * a.iz;
    float* out = a.out + (size_t)blockIdx.x * n;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int y = warp; y < a.ny; y += kPlaneThreads / 32)
        for (int x = lane; x < a.nx; x += 32) sl[y * p + x] = __ldg(in + y * a.iy + x * a.ix);
    __syncthreads();
    for (int y = threadIdx.x; y < a.ny; y += kPlaneThreads) line_means(sl + y * p, so + y * p, a.nx, a.r, 1);
    __syncthreads();
    for (int x = threadIdx.x; x < a.nx; x += kPlaneThreads) line_means(so + x, sl + x, a.ny, a.r, p);
    __syncthreads();
    for (int y = warp; y < a.ny; y += kPlaneThreads / 32)
        for (int x = lane; x < a.nx; x += 32) out[y * a.nx + x] = sl[y * p + x];
}

// The same sliding sums with the lines staged through shared memory: a CTA takes kLines
// consecutive lines, loads them with coalesced requests (along the line when it is
// contiguous, across lines otherwise), walks its line in shared memory and stores the
// means back the same way. Shared memory: 2 * L * (kLines + 1) floats.
constexpr int kLines = 32;               // lines per CTA: ~5000 lines per pass at 144^3 -> 160 CTAs
constexpr int kLineThreads = 128;        // the load and store phases use four warps
constexpr int kLp = kLines + 1;
__global__ void __launch_bounds__(kLineThreads) k_box_line_smem(LineArgs a, int along) {
    extern __shared__ float sl[];
    float* so = sl + (size_t)a.L * kLp;
    __shared__ long ibase[kLines], obase[kLines];
    __shared__ unsigned shist[256];
    if (a.hist)
        for (int k = threadIdx.x; k < 256; k += kLineThreads) shist[k] = 0;
    const long lines = a.A * a.B, t0 = (long)blockIdx.x * kLines;
    const int tid = threadIdx.x;
    const int nl = (int)(lines - t0 < kLines ? lines - t0 : kLines);
    if (tid < nl) {
        const long t = t0 + tid, ai = t / a.B, bi = t - ai * a.B;
        ibase[tid] = ai * a.ia + bi * a.ib;
        obase[tid] = ai * a.oa + bi * a.ob;
    }
    __syncthreads();
    // contiguous lines: consecutive threads walk along a line (k = j*L + e); otherwise they
    // walk across lines (k = e*kLines + j), skipping the missing lines of the last CTA
    const unsigned L = (unsigned)a.L, total = along ? (unsigned)nl * L : (unsigned)kLines * L;
#pragma unroll 4
    for (unsigned k = tid; k < total; k += kLineThreads) {
        const unsigned j = along ? k / L : k % kLines, e = along ? k - (k / L) * L : k / kLines;
        if ((int)j < nl) sl[e * kLp + j] = a.in[ibase[j] + (long)e * a.il];
    }
    __syncthreads();
    if (tid < nl) line_means(sl + tid, so + tid, a.L, a.r, kLp);
    __syncthreads();
#pragma unroll 4
    for (unsigned k = tid; k < total; k += kLineThreads) {
        const unsigned j = along ? k / L : k % kLines, e = along ? k - (k / L) * L : k / kLines;
        if ((int)j < nl) {
            const float v = so[e * kLp + j];
            a.out[obase[j] + (long)e * a.ol] = v;
            if (a.hist) {                   // pipeline.c:318-321: (int)(v*255 + 0.5), clamped
                int bin = (int)__fmaf_rn(v, 255.0f, 0.5f);
                bin = bin < 0 ? 0 : (bin > 255 ? 255 : bin);
                atomicAdd(&shist[bin], 1u);
            }
        }
    }
    if (a.hist) {
        __syncthreads();
        for (int k = threadIdx.x; k < 256; k += kLineThreads)
            if (shist[k]) atomicAdd(&a.hist[k], shist[k]);
    }
}

__global__ void __launch_bounds__(256) k_air_hist(const float* __restrict__ sm, size_t n, TileCtl* ctl) {
    __shared__ unsigned h[256];
    h[threadIdx.x] = 0;
    __syncthreads();
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        int b = (int)__fmaf_rn(sm[i], 255.0f, 0.5f);
        b = b < 0 ? 0 : (b > 255 ? 255 : b);
        atomicAdd(&h[b], 1u);
    }
    __syncthreads();
    if (h[threadIdx.x]) atomicAdd(&ctl->hist[threadIdx.x], h[threadIdx.x]);
}

// The valley (stream.c:138-168) and the value cut with its texture split (pipeline.c:330-378),
// one CTA of 256 threads, a thread per bin: smoothed counts, their maximum, the local-maximum
// candidates and the valley's first minimum in parallel; the peak merge, which is sequential
// by definition, walks the candidate bits on one thread. Same arithmetic as valley_depth_hd.
__global__ void __launch_bounds__(256) k_air_cut(TileCtl* ctl, int air_cut_u8, int air_cut_band, double air_thresh,
                                                 double air_cut_aggr) {
    __shared__ double hf[256];
    __shared__ double wmax[8];
    __shared__ unsigned cand[8];
    __shared__ int s_ab[3];
    __shared__ double wmin[8];
    __shared__ int wmini[8];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    long sum = 0;
    int cnt = 0;
    for (int j = t - 2; j <= t + 2; j++)
        if (j >= 0 && j < 256) { sum += ctl->hist[j]; cnt++; }
    double h = (double)sum / cnt;
    if (t == 0 || t == 254 || t == 255) h = 0;
    hf[t] = h;
    double m = h;
    for (int o = 16; o; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) wmax[warp] = m;
    __syncthreads();
    double mx = wmax[0];
    for (int k = 1; k < 8; k++) mx = fmax(mx, wmax[k]);
    const bool c = t >= 3 && t < 253 && hf[t] >= hf[t - 1] && hf[t] >= hf[t + 1] && hf[t] > 0.05 * mx;
    const unsigned bal = __ballot_sync(0xffffffffu, c);
    if (lane == 0) cand[warp] = bal;
    __syncthreads();
    if (t == 0) {
        int ok = 0, a = 0, b = 0;
        if (mx > 0) {
            int pk[32], np = 0;           // kept peaks are > 10 bins apart: at most 23 in [3, 253)
            for (int w = 0; w < 8; w++)
                for (unsigned bits = cand[w]; bits; bits &= bits - 1) {
                    const int u = w * 32 + __ffs(bits) - 1;
                    if (np > 0 && u - pk[np - 1] <= 10) {
                        if (hf[u] > hf[pk[np - 1]]) pk[np - 1] = u;
                    } else if (np < 32) {
                        pk[np++] = u;
                    }
                }
            if (np >= 2) {
                int p1 = pk[0], p2 = pk[1];
                for (int i = 0; i < np; i++) {
                    const int u = pk[i];
                    if (hf[u] > hf[p1]) { p2 = p1; p1 = u; }
                    else if (hf[u] > hf[p2] && u != p1) p2 = u;
                }
                a = p1 < p2 ? p1 : p2;
                b = p1 < p2 ? p2 : p1;
                ok = 1;
            }
        }
        s_ab[0] = a; s_ab[1] = b; s_ab[2] = ok;
    }
    __syncthreads();
    const int a = s_ab[0], b = s_ab[1], ok = s_ab[2];
    // first minimum over [a, b] (strict <, so the lowest bin among equal minima)
    double vm = (ok && t >= a && t <= b) ? hf[t] : INFINITY;
    int vi = (ok && t >= a && t <= b) ? t : 1 << 30;
    for (int o = 16; o; o >>= 1) {
        const double ov = __shfl_xor_sync(0xffffffffu, vm, o);
        const int oi = __shfl_xor_sync(0xffffffffu, vi, o);
        if (ov < vm || (ov == vm && oi < vi)) { vm = ov; vi = oi; }
    }
    if (lane == 0) { wmin[warp] = vm; wmini[warp] = vi; }
    __syncthreads();
    if (t != 0) return;
    int dark = 0, light = 0, valley = 0;
    double d = -1;
    if (ok) {
        double vmin = wmin[0];
        int v = wmini[0];
        for (int k = 1; k < 8; k++)
            if (wmin[k] < vmin || (wmin[k] == vmin && wmini[k] < v)) { vmin = wmin[k]; v = wmini[k]; }
        dark = a; light = b; valley = v;
        const double mn = hf[a] < hf[b] ? hf[a] : hf[b];
        d = 1.0 - vmin / (mn + 1e-12);
    }
    const int pf = air_thresh > 0 ? (int)__fma_rn(air_thresh, 255.0, 0.5) : 39;
    int cut;
    if (air_cut_u8 >= 0) {
        const int gg = air_cut_u8, band = air_cut_band;
        if (d >= 0) {
            double g = air_cut_aggr;
            g = g < 0 ? 0 : (g > 2 ? 2 : g);
            int local;
            if (valley <= pf) local = pf;
            else if (g <= 1.0) local = (int)__dadd_rn(__fma_rn(g, (double)(valley - pf), (double)pf), 0.5);
            else
                local = (int)__dadd_rn(
                    __fma_rn(__dsub_rn(g, 1.0), (double)(light > valley ? light - valley : 0), (double)valley), 0.5);
            cut = local < gg - band ? gg - band : (local > gg + band ? gg + band : local);
        } else {
            cut = gg;
        }
    } else if (d >= 0) {
        const int mid = (dark + valley) / 2;
        cut = dark + 8 < mid ? dark + 8 : mid;
    } else {
        cut = (int)__dmul_rn(air_thresh > 0 ? air_thresh : 0.05, 255.0);
    }
    const int spread = valley > pf ? (valley - pf) / 2 : 8;
    int cu = cut + spread;
    if (valley > cut && cu > valley) cu = valley;
    int ct = cut - spread;
    if (ct < pf) ct = pf;
    ctl->cuts[0] = cut;
    ctl->cuts[1] = cu;
    ctl->cuts[2] = ct;
    ctl->cutf_uni = __fmul_rn((float)cu, 1.0f / 255.0f);
    ctl->cutf_tex = __fmul_rn((float)ct, 1.0f / 255.0f);
}

// Rows (x lines) taken by one CTA of the row kernels: a warp each, no barrier.
constexpr int kRowWarps = 8;

struct AirArgs {
    float* f;                 // may alias orig: each voxel reads orig and writes f at itself
    const float* orig;
    const float* sm;
    const TileCtl* ctl;
    long nz, ny, nx, lz, ly, lx;
    int lowres;
    unsigned* mask;           // despeckle on: a bit per voxel, material (f > 0), rows of `words` words
    int words;
    int* lab;                 // despeckle on: parents of the run heads (k_cc_union's nodes)
    unsigned* info;
};

__device__ __forceinline__ float blend4(float s00, float s01, float s10, float s11, float w00, float w01, float w10,
                                        float w11) {
    return __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(w00, s00), __fmul_rn(w01, s01)), __fmul_rn(w10, s10)),
                     __fmul_rn(w11, s11));
}

// zero f where the scratch smooth (trilinear from the decimated grid) is below the cut,
// the cut chosen by the local texture |orig - smooth| (pipeline.c:355-399).
//
// Bound by issue and latency, not by memory (the fields of a tile live in L2): a warp takes a whole
// row, so that everything of y and z is formed once per row, and walks it 32 voxels at a time. The
// material bits come out of the walk's ballots, and with the run carried from word to word each
// word's first voxel can point at its run's head in an earlier word: no barrier, and labels only at
// run heads instead of at every voxel. Measured at 144^3:
// 21.9 us against 31.8 with a CTA per row, which also wrote a label per voxel.
__global__ void __launch_bounds__(32 * kRowWarps) k_air_apply(AirArgs a) {
    const unsigned row = blockIdx.x * kRowWarps + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31, nx = (int)a.nx;
    if (row >= (unsigned)(a.nz * a.ny)) return;
    const int z = (int)(row / (unsigned)a.ny), y = (int)(row - (unsigned)z * (unsigned)a.ny);
    const float cu = a.ctl->cutf_uni, ct = a.ctl->cutf_tex;
    const int base = (int)(row * (unsigned)nx);
    int z0 = z >> 1, y0 = y >> 1;
    if (z0 > a.lz - 2) z0 = (int)a.lz - 2;
    if (y0 > a.ly - 2) y0 = (int)a.ly - 2;
    float zf = __fsub_rn(__fmul_rn(0.5f, (float)z), (float)z0), yf = __fsub_rn(__fmul_rn(0.5f, (float)y), (float)y0);
    zf = zf > 1.0f ? 1.0f : zf;
    yf = yf > 1.0f ? 1.0f : yf;
    const float w00 = __fmul_rn(1.0f - zf, 1.0f - yf), w01 = __fmul_rn(1.0f - zf, yf);
    const float w10 = __fmul_rn(zf, 1.0f - yf), w11 = __fmul_rn(zf, yf);
    const int lx = (int)a.lx;
    const float* s00 = a.sm + (a.lowres ? ((size_t)z0 * a.ly + y0) * lx : (size_t)base);
    const float *s01 = s00 + lx, *s10 = s00 + (size_t)a.ly * lx, *s11 = s10 + lx;
    int head = -1;                           // first voxel of the run that reaches the word's end, or -1
    for (int w = 0; w * 32 < nx; ++w) {
        const int x = w * 32 + lane;
        bool mat = false;
        if (x < nx) {
            float v;
            if (a.lowres) {
                int x0 = x >> 1;
                if (x0 > lx - 2) x0 = lx - 2;
                float fx = __fsub_rn(__fmul_rn(0.5f, (float)x), (float)x0);
                fx = fx > 1.0f ? 1.0f : fx;
                const float a0 = blend4(s00[x0], s01[x0], s10[x0], s11[x0], w00, w01, w10, w11);
                const float a1 = blend4(s00[x0 + 1], s01[x0 + 1], s10[x0 + 1], s11[x0 + 1], w00, w01, w10, w11);
                v = __fmaf_rn(__fsub_rn(a1, a0), fx, a0);
            } else {
                v = s00[x];
            }
            const float tex = fabsf(__fsub_rn(a.orig[base + x], v));
            const float fv = a.f[base + x];
            const bool air = v < (tex < 0.03f ? cu : ct);
            if (air) a.f[base + x] = 0.0f;
            mat = !air && fv > 0.0f;
        }
        if (a.mask) {
            const unsigned bits = __ballot_sync(0xffffffffu, mat);
            if (mat && (lane == 0 || !(bits >> (lane - 1) & 1u))) {
                a.lab[base + x] = lane == 0 && head >= 0 ? head : base + x;
                a.info[base + x] = 0u;
            }
            if (lane == 0) a.mask[(size_t)row * a.words + w] = bits;
            if (!(bits >> 31)) head = -1;
            else if (~bits) head = base + w * 32 + 32 - __clz(~bits);
            else if (head < 0) head = base + w * 32;
        }
    }
}

// ---------------------------------------------------------------- connected components
__device__ __forceinline__ int uf_find(int* L, int i, int* err) {
    for (int it = 0; it < kUfMaxIter; ++it) {
        const int p = __ldcg(L + i);     // L2 reads: links made by other threads are seen
        if (p == i) return i;
        const int g = __ldcg(L + p);
        if (g != p) L[i] = g;            // path halving: g is an ancestor of i
        i = g;
    }
    *err = 1;
    return i;
}

// Read-only walk to the root: the flatten pass uses it, so that no store of another walk can
// land on a label after its final root was written.
__device__ __forceinline__ int uf_root(const int* L, int i, int* err) {
    for (int it = 0; it < kUfMaxIter; ++it) {
        const int p = __ldcg(L + i);
        if (p == i) return i;
        i = p;
    }
    *err = 1;
    return i;
}

__device__ __forceinline__ void uf_union(int* L, int a, int b, int* err) {
    for (int it = 0; it < kUfMaxIter; ++it) {
        a = uf_find(L, a, err);
        b = uf_find(L, b, err);
        if (a == b) return;
        if (a < b) { const int t = a; a = b; b = t; }   // link the larger root under the smaller
        const int old = atomicMin(&L[a], b);
        if (old == a) return;
        a = old;
    }
    *err = 1;
}

struct CcArgs {
    const unsigned* mask;
    int words;
    int* lab;
    unsigned* info;
    int* err;
    int nz, ny, nx;
    int min_size;
};

// The nodes of the union-find are the x-runs of material within a word of 32 voxels, each named by
// its first voxel; a run that enters a word from the left was linked to its head by the air pass.
// The run of bit b of word c starts at:
__device__ __forceinline__ int run_start(unsigned c, int b) {
    const unsigned gaps = ~c & ((1u << b) - 1u);
    return gaps ? 32 - __clz(gaps) : 0;
}

// Join runs to those of the -y (blockIdx.y = 0) and -z (1) neighbour rows, once per overlap: where
// an overlap starts (if the left neighbours are both material, they already joined the runs). A
// thread takes a word, so that a solid row costs five threads and one join instead of a test of six
// labels at each of its voxels; what is left is the walks' latency. Measured at 144^3:
// 35.7 us against 39.7. (Joining blocks of rows in shared memory first cost more than it took off this
// pass: 29 us for the blocks, 9 to 20 us left here.)
__global__ void __launch_bounds__(128) k_cc_union(CcArgs a) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (unsigned)a.nz * a.ny * a.words) return;
    const unsigned row = t / (unsigned)a.words, w = t - row * (unsigned)a.words;
    const unsigned z = row / (unsigned)a.ny, y = row - z * (unsigned)a.ny;
    const unsigned back = blockIdx.y ? (unsigned)a.ny : 1u;          // rows to the neighbour
    if (blockIdx.y ? z == 0 : y == 0) return;
    const unsigned q = t - back * (unsigned)a.words;
    const unsigned c = a.mask[t], u = a.mask[q], o = c & u;
    if (!o) return;
    const unsigned joined = w ? (a.mask[t - 1] & a.mask[q - 1]) >> 31 : 0u;
    const int i = (int)(row * (unsigned)a.nx + w * 32u), j = i - (int)(back * (unsigned)a.nx);
    for (unsigned s = o & ~(o << 1 | joined); s; s &= s - 1) {
        const int b = __ffs(s) - 1;
        uf_union(a.lab, i + run_start(c, b), j + run_start(u, b), a.err);
    }
}

// Roots by read-only walks from the nodes (stored for the quantiser), component sizes and face
// contact. A count stops growing once it reaches min_size and a face-touching root takes no count:
// both leave the zero test (no face contact and fewer than min_size voxels) unchanged, and a root
// already known to be either takes no more atomics (the giant components would otherwise serialise
// on one address). A thread takes a word and adds up its runs of one root; the last root of each
// thread is added up over the warp. Measured at 144^3: 16.0 us against 29.1 with a thread per
// voxel.
__global__ void __launch_bounds__(128) k_cc_count(CcArgs a) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    auto put = [&](int root, unsigned n, unsigned edge) {
        const unsigned v = __ldcg(a.info + root);
        if (v & kEdge) return;
        if (edge) atomicOr(&a.info[root], kEdge);
        else if ((long)v < a.min_size) atomicAdd(&a.info[root], n);
    };
    int cur = -1;
    unsigned n = 0, edge = 0;
    if (t < (unsigned)a.nz * a.ny * a.words) {
        const unsigned row = t / (unsigned)a.words, w = t - row * (unsigned)a.words;
        const int z = (int)(row / (unsigned)a.ny), y = (int)(row - (unsigned)z * (unsigned)a.ny);
        const bool face = z == 0 || z == a.nz - 1 || y == 0 || y == a.ny - 1;
        const int i = (int)(row * (unsigned)a.nx + w * 32u);
        unsigned c = a.mask[t];
        while (c) {
            const int b = __ffs(c) - 1;
            const unsigned gaps = ~(c >> b);                         // shifted-in zeros are gaps
            const int len = gaps ? __ffs(gaps) - 1 : 32;
            c = b + len < 32 ? c & ~((1u << (b + len)) - 1u) : 0u;
            const int root = uf_root(a.lab, i + b, a.err);
            a.lab[i + b] = root;
            const unsigned e = face || (w == 0 && b == 0) || (int)w * 32 + b + len == a.nx;
            if (root != cur) {
                if (cur >= 0) put(cur, n, edge);
                cur = root; n = 0; edge = 0;
            }
            n += len;
            edge |= e;
        }
    }
    const unsigned peers = __match_any_sync(0xffffffffu, cur);
    n = __reduce_add_sync(peers, n);
    edge = __reduce_or_sync(peers, edge);
    if (cur >= 0 && __ffs(peers) - 1 == (int)(threadIdx.x & 31)) put(cur, n, edge);
}

// ---------------------------------------------------------------- recenter + quantise
struct QuantArgs {
    const float* f;
    uint8_t* out;
    long hy, hx;
    long iz0, iy0, ix0;       // inner tile origin inside the buffer
    long tz, ty, tx;
    long gz0, gy0, gx0;       // inner tile origin in the volume
    int no_dither, norm;
    float midf, k;
    const unsigned* mask;     // despeckle on: material bits, else nullptr
    int words;
    const int* lab;           // run head -> component root (k_cc_count)
    const unsigned* info;
    int min_size;
};

// A warp per row of the inner tile. Measured at 128^3 inside 144^3: 12.6 us against 15.3 with a CTA per
// row and a label per voxel.
__global__ void __launch_bounds__(32 * kRowWarps) k_tile_quant(QuantArgs a) {
    const unsigned row = blockIdx.x * kRowWarps + (threadIdx.x >> 5);
    if (row >= (unsigned)(a.tz * a.ty)) return;
    const int z = (int)(row / (unsigned)a.ty), y = (int)(row - (unsigned)z * (unsigned)a.ty);
    const size_t brow = (size_t)(a.iz0 + z) * a.hy + (a.iy0 + y);
    const float* f = a.f + brow * a.hx + a.ix0;
    const unsigned* mask = a.mask + (a.mask ? brow * a.words : 0);
    uint8_t* out = a.out + (size_t)row * a.tx;
    for (int x = (int)(threadIdx.x & 31); x < (int)a.tx; x += 32) {
        float v = f[x];
        if (a.mask) {                       // the despeckle's zeroing, for the voxels kept
            const int bx = (int)a.ix0 + x, b = bx & 31;
            const unsigned c = mask[bx >> 5];
            if (c >> b & 1u) {
                const unsigned m = a.info[a.lab[brow * a.hx + (bx - b) + run_start(c, b)]];
                if (!(m & kEdge) && (long)m < a.min_size) v = 0.0f;
            }
        }
        if (a.norm) {
            if (v <= 0.0f) {
                v = 0.0f;
            } else {
                const float w = __fadd_rn(0.5f, __fmul_rn(__fsub_rn(v, a.midf), a.k));   // not fused, as the reference build
                v = w < 0.0f ? 0.0f : (w > 1.0f ? 1.0f : w);
            }
        }
        const float t = __fmaf_rn(v, 255.0f, a.no_dither ? 0.5f : dither01(a.gz0 + z, a.gy0 + y, a.gx0 + x));
        uint8_t q = 0;
        if (t > 0.0f) {
            const int qi = (int)t;
            q = qi > 255 ? 255 : (uint8_t)qi;
        }
        out[x] = q;
    }
}

// ---------------------------------------------------------------- host side
struct TileWs {
    fy::DevBuf u8, orig, work, alt, t1, t2, sm, mask, lab, info, tab, ctl, out;
    fy::HostBuf pin, hin, hout;   // control and tables; host-API staging of the u8 tile in/out
    bool have_state = false;
    long hist[256];
    int cuts[3];
};
thread_local TileWs tws;

unsigned grid1(size_t n, int tpb, int sms) {
    size_t g = (n + tpb - 1) / tpb, cap = (size_t)sms * 8;
    return (unsigned)std::max<size_t>(1, std::min(g, cap));
}

// Row kernels: a warp per row.
unsigned grid_rows(long ny, long nz) { return (unsigned)((ny * nz + kRowWarps - 1) / kRowWarps); }

// eps_for_tile, pipeline.c:447-456
double tile_eps(const fy_pipeline_cfg* c, double ecy, double ecx, long y0, long x0, long ty, long tx) {
    if (!c->have_eps_r || c->guided_eps <= 0 || c->eps_fn_med <= 0) return 0.0;
    const double ry = y0 + ty / 2.0 - ecy, rx = x0 + tx / 2.0 - ecx;
    const double fn = c->eps_fn_a + c->eps_fn_b * sqrt(ry * ry + rx * rx);
    const double s = fn / c->eps_fn_med;
    double s2 = s * s;
    if (s2 < 0.4) s2 = 0.4;
    if (s2 > 8.0) s2 = 8.0;
    return c->guided_eps * s2;
}

// One pass of line sums; with ctl set (the last pass) the histogram of the means is added
// to ctl->hist as they are stored (or by k_air_hist after the unstaged kernel).
cudaError_t box_pass(const float* in, float* out, int L, int r, long A, long B, long ia, long ib, long il, long oa,
                     long ob, long ol, cudaStream_t st, TileCtl* ctl = nullptr, int sms = 148) {
    LineArgs a{in, out, L, r, A, B, ia, ib, il, oa, ob, ol, nullptr};
    const long lines = A * B;
    const size_t smem = (size_t)2 * L * kLp * sizeof(float);
    if (smem <= 200 * 1024) {
        cudaError_t e = fy_smem_optin(k_box_line_smem, smem);
        if (e != cudaSuccess) return e;
        a.hist = ctl ? ctl->hist : nullptr;
        k_box_line_smem<<<(unsigned)((lines + kLines - 1) / kLines), kLineThreads, smem, st>>>(a, ib != 1 ? 1 : 0);
    } else {
        k_box_line<<<(unsigned)((lines + kTpb - 1) / kTpb), kTpb, 0, st>>>(a);
        if (ctl) {
            const size_t m = (size_t)A * B * L;
            k_air_hist<<<grid1(m, 256, sms), 256, 0, st>>>(out, m, ctl);
        }
    }
    return cudaGetLastError();
}

#define TRY(call)                                           \
    do {                                                    \
        cudaError_t e_ = (call);                            \
        if (e_ != cudaSuccess) return fail_cuda(e_, what);  \
    } while (0)

int tile_chain(const fy_pipeline_cfg* c, const uint8_t* d_u8, long rz0, long ry0, long rx0, long hz, long hy,
               long hx, long z0, long y0, long x0, long tz, long ty, long tx, long vol_y, long vol_x, uint8_t* d_out,
               int* all_air, cudaStream_t st, const char* what) {
    fy::ThreadCtx& cx = ctx();
    TileWs& w = tws;
    w.have_state = false;
    const size_t hn = (size_t)hz * hy * hx, tn = (size_t)tz * ty * tx;
    TRY(w.ctl.ensure(sizeof(TileCtl)));
    TRY(w.pin.ensure(sizeof(TileCtl)));
    TileCtl* ctl = w.ctl.as<TileCtl>();
    TileCtl* hctl = (TileCtl*)w.pin.p;
    TRY(cudaMemsetAsync(ctl, 0, sizeof(TileCtl), st));
    k_tile_any<<<grid1(hn / 16 + 1, 256, cx.sms), 256, 0, st>>>(d_u8, hn, ctl);
    TRY(cudaGetLastError());
    TRY(cudaMemcpyAsync(hctl, ctl, sizeof(int) * 2, cudaMemcpyDeviceToHost, st));
    TRY(cudaStreamSynchronize(st));
    int launches = 1;
    if (!hctl->any) {
        if (tn) TRY(cudaMemsetAsync(d_out, 0, tn, st));
        TRY(cudaStreamSynchronize(st));
        fy::count_launch(launches);
        if (all_air) *all_air = 1;
        return FY_OK;
    }
    if (c->do_musica) return fail(FY_EUNSUPPORTED, "%s: MUSICA is not on the GPU path", what);

    // ring rows and z-drift factors of this buffer, staged through pinned memory
    const fy_dering* dr = c->have_dering ? c->dering : nullptr;
    const bool rings = dr && dr->have_rings && dr->ring && dr->nr > 0 && dr->nslab > 0 && dr->slab_z > 0;
    const bool zdrift = c->have_zdrift && c->zdrift_factor;
    long s0 = 0, s1 = -1;
    if (rings) {
        auto slab = [&](long z) { long s = z / dr->slab_z; return s < 0 ? 0L : (s >= dr->nslab ? (long)dr->nslab - 1 : s); };
        s0 = slab(rz0);
        s1 = slab(rz0 + hz - 1);
    }
    const size_t ring_floats = rings ? (size_t)(s1 - s0 + 1) * dr->nr : 0, zd_floats = zdrift ? (size_t)hz : 0;
    const size_t ctl_bytes = (sizeof(TileCtl) + 255) & ~(size_t)255;
    const size_t tab_bytes = (ring_floats + zd_floats) * sizeof(float);
    const float* d_ring = nullptr;
    const float* d_zd = nullptr;
    if (tab_bytes) {
        TRY(w.pin.ensure(ctl_bytes + tab_bytes));
        hctl = (TileCtl*)w.pin.p;
        float* h = (float*)((char*)w.pin.p + ctl_bytes);
        if (rings) memcpy(h, dr->ring + (size_t)s0 * dr->nr, ring_floats * sizeof(float));
        if (zdrift) memcpy(h + ring_floats, c->zdrift_factor + rz0, zd_floats * sizeof(float));
        TRY(w.tab.ensure(tab_bytes));
        TRY(cudaMemcpyAsync(w.tab.p, h, tab_bytes, cudaMemcpyHostToDevice, st));
        if (rings) d_ring = w.tab.as<float>();
        if (zdrift) d_zd = w.tab.as<float>() + ring_floats;
    }

    // Buffers: orig (the pre-deconvolution copy) always; the working field is orig itself
    // until a stage writes a new one (deconvolution in place on `work`, guided into `alt`),
    // since the air cut reads orig and writes f one voxel at a time.
    TRY(w.orig.ensure(hn * sizeof(float)));
    float* orig = w.orig.as<float>();
    float* f = orig;
    if (c->do_deconv) {
        TRY(w.work.ensure(hn * sizeof(float)));
        f = w.work.as<float>();
    }
    const bool windowed = c->window_hi > c->window_lo;
    const float wlo = (float)c->window_lo, wspan = (float)(c->window_hi - c->window_lo);
    {
        PrepArgs a{};
        a.u8 = d_u8; a.orig = orig; a.work = c->do_deconv ? f : nullptr;
        a.hz = hz; a.hy = hy; a.hx = hx;
        a.ring = d_ring;
        if (rings) {
            a.s0 = s0; a.nslab = dr->nslab; a.slab_z = dr->slab_z; a.nr = dr->nr; a.cy = dr->cy; a.cx = dr->cx;
        } else {
            a.slab_z = 1; a.nslab = 1;
        }
        a.rz0 = rz0; a.ry0 = ry0; a.rx0 = rx0;
        a.sc = (float)(1.0 / 255.0);
        a.zdrift = d_zd;
        a.windowed = c->do_deconv && windowed;
        a.wlo = wlo; a.wspan = wspan;
        k_tile_prep<<<grid1((hn + 3) / 4, 256, cx.sms), 256, 0, st>>>(a);
        TRY(cudaGetLastError());
        launches++;
        fy_prof_mark(st, "tile.prep");
    }

    int rc;
    if (c->do_deconv) {                                           // pipeline.c:260-288
        fy_physics ph{c->delta_beta, c->energy_kev, c->distance_mm, c->pixel_um, c->unsharp_sigma, c->unsharp_coeff,
                      c->psf_sigma_vox,
                      (c->psf_z_ratio > 1.0 && c->psf_sigma_vox > 0) ? c->psf_z_ratio * c->psf_sigma_vox : 0.0};
        ph.delta_beta *= fy_auto_deltabeta_scale(&ph);
        const bool matched = c->use_matched_deconv && c->psf_sigma_vox > 0;
        if ((rc = fy_gpu_deconvolve_ex(f, 0, 0.0, 0.0, f, (int)hz, (int)hy, (int)hx, &ph,
                                       matched ? c->deconv_tikhonov : -1.0, matched ? 1 : 0, 1.0, st)))
            return rc;
        const bool rescale = c->have_dec_range && c->dec_hi - c->dec_lo > 1e-6;
        k_tile_unwin<<<grid1(hn, 256, cx.sms), 256, 0, st>>>(f, hn, windowed, wlo, windowed ? 1.0f / wspan : 1.0f,
                                                             rescale, (float)c->dec_lo,
                                                             rescale ? 1.0f / (float)(c->dec_hi - c->dec_lo) : 1.0f);
        TRY(cudaGetLastError());
        launches++;
        fy_prof_mark(st, "tile.unwin");
    }

    const double ecy = c->dering_cy > 0 ? c->dering_cy : (vol_y - 1) / 2.0;
    const double ecx = c->dering_cx > 0 ? c->dering_cx : (vol_x - 1) / 2.0;
    const double teps = tile_eps(c, ecy, ecx, y0, x0, ty, tx);
    if (c->guided_eps > 0 || teps > 0) {                          // pipeline.c:290-297
        const double eps = teps > 0 ? teps : c->guided_eps;
        const int gs = c->guided_subsample == 0 ? 2 : c->guided_subsample;
        TRY(w.alt.ensure(hn * sizeof(float)));
        float* g = w.alt.as<float>();
        if ((rc = fy_gpu_guided(f, g, (int)hz, (int)hy, (int)hx, 2, eps, gs, st))) return rc;
        f = g;
        fy_prof_mark(st, "tile.guided");
    }

    if (c->do_air_zero) {                                         // pipeline.c:299-405
        const int sr = c->scratch_passes > 0 ? c->scratch_passes : 5;
        const long lz = (hz + 1) / 2, ly = (hy + 1) / 2, lx = (hx + 1) / 2;
        const bool lowres = lz >= 2 && ly >= 2 && lx >= 2;
        const long mz = lowres ? lz : hz, my = lowres ? ly : hy, mx = lowres ? lx : hx;
        const size_t m = (size_t)mz * my * mx;
        const int r = lowres ? std::max(1, (sr + 1) / 2) : sr;
        const long d = lowres ? 2 : 1;
        TRY(w.t2.ensure(m * sizeof(float)));
        TRY(w.sm.ensure(m * sizeof(float)));
        float *t2 = w.t2.as<float>(), *sm = w.sm.as<float>();
        const long mp = my * mx;
        // x lines (decimated read of orig), then y lines, then z lines
        const size_t plane_smem = (size_t)2 * my * (mx | 1) * sizeof(float);
        if (plane_smem <= 200 * 1024) {
            TRY(fy_smem_optin(k_box_plane, plane_smem));
            PlaneArgs pa{orig, t2, (int)my, (int)mx, r, d * hy * hx, d * hx, d};
            k_box_plane<<<(unsigned)mz, kPlaneThreads, plane_smem, st>>>(pa);
            TRY(cudaGetLastError());
            launches--;
        } else {
            TRY(w.t1.ensure(m * sizeof(float)));
            float* t1 = w.t1.as<float>();
            TRY(box_pass(orig, t1, (int)mx, r, mz, my, d * hy * hx, d * hx, d, mp, mx, 1, st));
            TRY(box_pass(t1, t2, (int)my, r, mz, mx, mp, 1, mx, mp, 1, mx, st));
        }
        TRY(box_pass(t2, sm, (int)mz, r, my, mx, mx, 1, mp, mx, 1, mp, st, ctl, cx.sms));   // + histogram
        fy_prof_mark(st, "tile.scratch_box");
        k_air_cut<<<1, 256, 0, st>>>(ctl, c->air_cut_u8, c->air_cut_band, c->air_thresh, c->air_cut_aggr);
        TRY(cudaGetLastError());
        fy_prof_mark(st, "tile.air_cut");
        const bool cc = c->air_min_component > 0;
        const int words = (int)((hx + 31) / 32);
        const size_t nwords = (size_t)hz * hy * words;
        if (cc) {
            TRY(w.mask.ensure(nwords * sizeof(unsigned)));
            TRY(w.lab.ensure(hn * sizeof(int)));
            TRY(w.info.ensure(hn * sizeof(unsigned)));
        }
        AirArgs aa{f, orig, sm, ctl, hz, hy, hx, lz, ly, lx, lowres ? 1 : 0, cc ? w.mask.as<unsigned>() : nullptr,
                   words, w.lab.as<int>(), w.info.as<unsigned>()};
        k_air_apply<<<grid_rows(hy, hz), 32 * kRowWarps, 0, st>>>(aa);
        TRY(cudaGetLastError());
        launches += 5;
        fy_prof_mark(st, "tile.air_apply");
        if (cc) {
            CcArgs ca{w.mask.as<unsigned>(), words, w.lab.as<int>(), w.info.as<unsigned>(), &ctl->err,
                      (int)hz, (int)hy, (int)hx, c->air_min_component};
            const unsigned cg = (unsigned)((nwords + 127) / 128);
            k_cc_union<<<dim3(cg, 2), 128, 0, st>>>(ca);
            fy_prof_mark(st, "tile.cc_union");
            k_cc_count<<<cg, 128, 0, st>>>(ca);
            TRY(cudaGetLastError());
            launches += 2;
            fy_prof_mark(st, "tile.cc_count");
            // the zeroing of small interior components happens in the quantiser, which
            // reads the inner tile only
        }
    }

    {                                                             // pipeline.c:407-421, 500-506
        QuantArgs q{};
        q.f = f; q.out = d_out; q.hy = hy; q.hx = hx;
        q.iz0 = z0 - rz0; q.iy0 = y0 - ry0; q.ix0 = x0 - rx0;
        q.tz = tz; q.ty = ty; q.tx = tx;
        q.gz0 = z0; q.gy0 = y0; q.gx0 = x0;
        q.no_dither = c->no_dither;
        q.norm = c->have_norm && c->norm_hi > c->norm_lo;
        q.midf = 0.5f * (float)(c->norm_lo + c->norm_hi) * (1.0f / 255.0f);
        q.k = q.norm ? (2.0f * 0.375f) * 255.0f / (float)(c->norm_hi - c->norm_lo) : 0.0f;
        const bool cc = c->do_air_zero && c->air_min_component > 0;
        q.mask = cc ? w.mask.as<unsigned>() : nullptr;
        q.words = (int)((hx + 31) / 32);
        q.lab = w.lab.as<int>();
        q.info = w.info.as<unsigned>();
        q.min_size = c->air_min_component;
        if (tn) {
            k_tile_quant<<<grid_rows(ty, tz), 32 * kRowWarps, 0, st>>>(q);
            TRY(cudaGetLastError());
            launches++;
        }
        fy_prof_mark(st, "tile.quant");
    }
    TRY(cudaMemcpyAsync(hctl, ctl, sizeof(TileCtl), cudaMemcpyDeviceToHost, st));
    TRY(cudaStreamSynchronize(st));
    fy::count_launch(launches);
    if (hctl->err) return fail(FY_ETIMEDOUT, "%s: connected-component walk exceeded %d steps", what, kUfMaxIter);
    if (c->do_air_zero) {
        for (int i = 0; i < 256; i++) w.hist[i] = hctl->hist[i];
        for (int i = 0; i < 3; i++) w.cuts[i] = hctl->cuts[i];
        w.have_state = true;
    }
    if (all_air) *all_air = 0;
    return FY_OK;
}

int check_geometry(const fy_pipeline_cfg* c, const void* in, const void* out, long rz0, long ry0, long rx0, long hz,
                   long hy, long hx, long z0, long y0, long x0, long tz, long ty, long tx, const char* what) {
    if (!c || !in || !out) return fail(FY_EINVAL, "%s: null pointer", what);
    if (hz < 1 || hy < 1 || hx < 1 || tz < 0 || ty < 0 || tx < 0)
        return fail(FY_EINVAL, "%s: bad dims %ldx%ldx%ld / %ldx%ldx%ld", what, hz, hy, hx, tz, ty, tx);
    if (z0 < rz0 || y0 < ry0 || x0 < rx0 || z0 + tz > rz0 + hz || y0 + ty > ry0 + hy || x0 + tx > rx0 + hx)
        return fail(FY_EINVAL, "%s: inner tile outside the buffer", what);
    if ((double)hz * hy * hx >= 2147483647.0 || hy > 65535 || ty > 65535)
        return fail(FY_EUNSUPPORTED, "%s: buffer %ldx%ldx%ld too large for one tile", what, hz, hy, hx);
    if (c->do_deconv && (hz > INT32_MAX || hy > INT32_MAX || hx > INT32_MAX))
        return fail(FY_EUNSUPPORTED, "%s: dims", what);
    return FY_OK;
}

}  // namespace

extern "C" double fy_valley_depth(const long hist[256], int* dark_out, int* light_out, int* valley_out) {
    return valley_depth_hd(hist, dark_out, light_out, valley_out);
}

extern "C" int fy_gpu_process_buffer(const fy_pipeline_cfg* cfg, const unsigned char* d_u8, long rz0, long ry0,
                                     long rx0, long hz, long hy, long hx, long z0, long y0, long x0, long tz, long ty,
                                     long tx, long vol_y, long vol_x, unsigned char* d_out, int* all_air,
                                     void* stream) {
    fy::enter();
    const char* what = "fy_gpu_process_buffer";
    int rc = check_geometry(cfg, d_u8, d_out, rz0, ry0, rx0, hz, hy, hx, z0, y0, x0, tz, ty, tx, what);
    if (rc) return rc;
    if ((rc = fy::ensure_ctx())) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    fy::ws_acquire(st);
    rc = tile_chain(cfg, d_u8, rz0, ry0, rx0, hz, hy, hx, z0, y0, x0, tz, ty, tx, vol_y, vol_x, d_out, all_air, st,
                    what);
    fy::ws_release(st);
    return rc;
}

extern "C" int fy_process_buffer(const fy_pipeline_cfg* cfg, const unsigned char* u8buf, long rz0, long ry0,
                                 long rx0, long hz, long hy, long hx, long z0, long y0, long x0, long tz, long ty,
                                 long tx, long vol_y, long vol_x, unsigned char* out, int* all_air) {
    fy::enter();
    const char* what = "fy_process_buffer";
    int rc = check_geometry(cfg, u8buf, out, rz0, ry0, rx0, hz, hy, hx, z0, y0, x0, tz, ty, tx, what);
    if (rc) return rc;
    if ((rc = fy::ensure_ctx())) return rc;
    fy::ThreadCtx& c = ctx();
    cudaStream_t st = c.st;
    TileWs& w = tws;
    const size_t hn = (size_t)hz * hy * hx, tn = (size_t)tz * ty * tx;
    fy::ws_acquire(st);
    cudaError_t e;
    if ((e = w.u8.ensure(hn)) != cudaSuccess || (e = w.out.ensure(tn ? tn : 1)) != cudaSuccess)
        return fail_cuda(e, what);
    // Pageable host buffers go through this thread's pinned staging, so that the copies are
    // plain DMA and the threads of a worker pool do not serialise on the driver's staging.
    const bool pin_in = fy::is_pinned(u8buf), pin_out = fy::is_pinned(out);
    const void* src = u8buf;
    if (!pin_in) {
        if ((e = w.hin.ensure(hn)) != cudaSuccess) return fail_cuda(e, what);
        memcpy(w.hin.p, u8buf, hn);
        src = w.hin.p;
    }
    if ((e = cudaMemcpyAsync(w.u8.p, src, hn, cudaMemcpyHostToDevice, st)) != cudaSuccess) return fail_cuda(e, what);
    rc = tile_chain(cfg, w.u8.as<uint8_t>(), rz0, ry0, rx0, hz, hy, hx, z0, y0, x0, tz, ty, tx, vol_y, vol_x,
                    w.out.as<uint8_t>(), all_air, st, what);
    if (rc) return rc;
    if (tn) {
        void* dst = out;
        if (!pin_out) {
            if ((e = w.hout.ensure(tn)) != cudaSuccess) return fail_cuda(e, what);
            dst = w.hout.p;
        }
        if ((e = cudaMemcpyAsync(dst, w.out.p, tn, cudaMemcpyDeviceToHost, st)) != cudaSuccess) return fail_cuda(e, what);
        if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return fail_cuda(e, what);
        if (!pin_out) memcpy(out, w.hout.p, tn);
    }
    fy::ws_release(st);
    return FY_OK;
}

void fy_tile_release() {
    TileWs& w = tws;
    for (fy::DevBuf* b : {&w.u8, &w.orig, &w.work, &w.alt, &w.t1, &w.t2, &w.sm, &w.mask, &w.lab, &w.info, &w.tab, &w.ctl, &w.out})
        b->release();
    w.pin.release();
    w.hin.release();
    w.hout.release();
    w.have_state = false;
}

extern "C" int fy_process_buffer_air_state(long hist[256], int cuts[3]) {
    const TileWs& w = tws;
    if (!w.have_state) return 1;
    if (hist) memcpy(hist, w.hist, sizeof w.hist);
    if (cuts) memcpy(cuts, w.cuts, sizeof w.cuts);
    return 0;
}
