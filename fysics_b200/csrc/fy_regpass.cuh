// fy_regpass.cuh -- the deconvolution's five passes for axis lengths with a register plan
// (fy_regfft.cuh).
#pragma once
#include <limits.h>
#include "fy_internal.h"
#include "fy_regfft.cuh"

namespace rf {

// ---------------------------------------------------------------- column passes (Y and Z)
// A CTA transforms W = 16 columns, one 128-byte run per point, with TPL threads a column, the
// column index fastest. Its tile crosses shared memory once per transform, stored point-major
// (s[i*W + l]: a half warp's 16 columns are 16 consecutive float2, no conflicts).
// What bounds them: HBM at 512 (the Y passes move 1.07 GB in 180 us, 0.91 of the measured copy
// rate), latency below. Sixteen warps an SM with 128 registers (16 bytes of spills at most): at 512^3
// the Z pass takes 313 us so; with its weight's position in 32 fraction bits it took 307, and in that
// form 379 us with 8-column tiles (64-byte runs) and 20 warps, 434 us with 24 warps at 80 registers
// (spills, and more tiles in flight than HBM serves well). The shared-memory passes that these replace
// took 237 (Y forward), 424 (Z) and 203 us (Y inverse) there; at 256^3 33, 57 and 27 us against 25, 37
// and 23 now.
template <int N> struct Col {
    static constexpr int W = 16, NT = W * tpl(N);
    static constexpr int warps = elems(N) <= 24 ? 24 : 16;
    static constexpr int minb = warps * 32 / NT;
    static constexpr int tile = N * W;                    // the exchange; the tail's twiddles follow
    static constexpr size_t smem = (size_t)(tile + Tail<N>::count) * sizeof(float2);
};

// The column of a thread. Columns kx < px/2 are taken W at a time from one row of the spectrum
// (plane p, stride pstride). The last one, kx = px/2, would cost a tile of its own per row with
// one column in W used (11% of the tiles at px = 256); instead W rows' last columns share a tile.
// Those tiles come first: their loads are 16 rows apart instead of one run and take longest.
// They take several times a regular tile's time (16 sectors a request), so they are made only where
// at least `least` regular tiles hide them; below that the partly filled tiles are faster. Measured
// (us, shared against own): Y at 16 x 384^2 26.8 / 10.3, 16 x 512^2 22.5 / 12.3, 64^3 8.2 / 6.3, 192^3
// 16.4 / 13.3, 256^3 26.6 / 28.6, 384^3 113 / 107, 512^3 190 / 179; Z at 128^3 14.3 / 12.3, 192^3
// 20.5 / 22.5, 256^3 36.9 / 38.9, 384^3 186 / 201, 512^3 305 / 311 (events around each pass). So a Y pass
// shares them from two waves of CTAs on up to 256 points (above, a tile of its own is under 5% more
// work), a Z pass from one. Phase correlation's passes always share (least = 0): of whole correlations,
// shared against own, single pairs of few rows lose (8 x 512^2 107 / 96 us, 64^3 67 / 61) and many rows or
// pairs gain (200^3 x 2 563 / 585, 64 pairs of 4 x 64^2 77 / 83).
struct ColTiles {
    int regular;              // tiles per row over the kx < px/2 columns (or over all hx columns)
    int rows;                 // rows (planes of a Y pass, y of a Z pass)
    unsigned last, total;     // tiles of last columns, tiles in all
    FastDiv dreg;
};
inline ColTiles col_tiles(int hx, int rows, int W, long least = 0) {
    ColTiles c;
    const bool split = hx > 1 && (hx - 1) % W == 0 && (long)((hx - 1) / W) * rows >= least;
    c.regular = split ? (hx - 1) / W : (hx + W - 1) / W;
    c.rows = rows;
    c.dreg = FastDiv((uint32_t)c.regular);
    c.last = split ? (unsigned)((rows + W - 1) / W) : 0u;
    c.total = (unsigned)c.regular * rows + c.last;
    return c;
}
struct Column {
    int kx, row;
    bool valid;
    FY_D Column(const ColTiles& c, int hx, int W, int l) {
        if (blockIdx.x >= c.last) {
            const unsigned b = blockIdx.x - c.last;
            row = (int)c.dreg.div(b);
            kx = (int)(b - (unsigned)row * c.regular) * W + l;
            valid = kx < hx;
        } else {
            row = (int)blockIdx.x * W + l;
            kx = hx - 1;
            valid = row < c.rows;
        }
    }
};

// Points i >= n of an axis padded to N are the reflected ones (paganin.c:121-128; N < 2n).
FY_D int pad_src(int i, int n) { return i < n ? i : 2 * n - 1 - i; }

template <int N, bool PAD>
FY_D void col_load(float2 (&v)[elems(N)], const float2* __restrict__ col, size_t es, int n, int t, bool valid) {
    const float2* p = col + (size_t)t * es;
    const size_t step = tpl(N) * es;
#pragma unroll
    for (int m = 0; m < elems(N); ++m) {
        if (PAD) {
            v[m] = valid ? col[(size_t)pad_src(t + tpl(N) * m, n) * es] : make_float2(0.f, 0.f);
        } else {
            v[m] = valid ? *p : make_float2(0.f, 0.f);
            p += step;
        }
    }
}
template <int N>
FY_D void col_store(const float2 (&v)[elems(N)], float2* __restrict__ col, size_t es, int n, int t, bool valid) {
    float2* p = col + (size_t)t * es;
    asm volatile("" : "+l"(p));       // the load's addresses are not kept across the transform
    const size_t step = tpl(N) * es;
#pragma unroll
    for (int m = 0; m < elems(N); ++m) {
        if (valid && t + tpl(N) * m < n) *p = v[m];
        p += step;
    }
}
template <int N, int SIGN>
FY_D void col_fft(float2 (&v)[elems(N)], float2* __restrict__ s, int l, int t) {
    using C = Col<N>;
    head<N, SIGN>(v);
    head_store<N>(v, t, [&](int b, int q, float2 x) { s[(b * head_len(N) + q) * C::W + l] = x; });
    __syncthreads();
#pragma unroll
    for (int m = 0; m < elems(N); ++m) v[m] = s[(t + tpl(N) * m) * C::W + l];
    tail<N, SIGN>(v, t, s + C::tile);
}

// Y pass over the stored planes: forward (SIGN -1; rows >= nin gathered by reflection) or inverse,
// storing rows < nout.
template <int N, int SIGN, bool PAD>
__global__ void __launch_bounds__(Col<N>::NT, Col<N>::minb)
k_col_y(float2* __restrict__ spec, SpecGeom g, const __grid_constant__ ColTiles ct, const float2* __restrict__ tw, int nin,
        int nout) {
    fy_pdl_wait();
    extern __shared__ float4 smem4[];
    constexpr int W = Col<N>::W;
    const int l = threadIdx.x % W, t = threadIdx.x / W;
    const Column c(ct, g.hx, W, l);
    float2* col = spec + (size_t)c.row * g.py * g.hxp + c.kx;
    float2* s = reinterpret_cast<float2*>(smem4);
    float2 v[elems(N)];
    col_load<N, PAD>(v, col, g.hxp, nin, t, c.valid);
    load_tail_twiddles<N>(s + Col<N>::tile, tw);          // the exchange's barrier covers them
    col_fft<N, SIGN>(v, s, l, t);
    col_store<N>(v, col, g.hxp, nout, t, c.valid);
}

// Z pass: forward (planes >= nz gathered by reflection), radial LUT weight, inverse, planes < nz stored.
// The forward transform ends on the points where the inverse begins, so the weight is applied in
// registers and the tile crosses shared memory twice in all (five times in the shared-memory
// kernel, which also copied its tables to every tile).
template <int N, bool PAD>
__global__ void __launch_bounds__(Col<N>::NT, Col<N>::minb)
k_col_z(float2* __restrict__ spec, SpecGeom g, const __grid_constant__ ColTiles ct, const float2* __restrict__ tw,
        const float* lut, const double* fz2, const double* __restrict__ fy2, const double* __restrict__ fx2, double us) {
    fy_pdl_wait();
    extern __shared__ float4 smem4[];
    constexpr int W = Col<N>::W;
    float2* s = reinterpret_cast<float2*>(smem4);
    const int l = threadIdx.x % W, t = threadIdx.x / W;
    const Column c(ct, g.hx, W, l);
    const size_t es = (size_t)g.py * g.hxp;
    float2* col = spec + (size_t)c.row * g.hxp + c.kx;
    float2 v[elems(N)];
    col_load<N, PAD>(v, col, es, g.nz, t, c.valid);
    load_tail_twiddles<N>(s + Col<N>::tile, tw);
    col_fft<N, -1>(v, s, l, t);
    asm volatile("" : "+l"(fz2), "+l"(lut));             // nor are the weights' loads moved before it
    // Table position p = (fz^2 + fy^2 + fx^2)*us of paganin.c:234-236, and its fraction, in FP64;
    // adding 2^52 towards zero leaves the integer part in the low word. The last point of the table,
    // p = 4096, is cell 4096, which the table continues with an equal entry.
    const double pyx = c.valid ? (__ldg(fy2 + c.row) + __ldg(fx2 + c.kx)) * us : 0.0;
#pragma unroll
    for (int m = 0; m < elems(N); ++m) {
        const double p = fma(__ldg(fz2 + t + tpl(N) * m), us, pyx), ip = __dadd_rz(p, 0x1p52);
        const float* cell = lut + min((unsigned)__double2loint(ip), (unsigned)FY_LUT_N);
        const float l0 = __ldg(cell), l1 = __ldg(cell + 1);
        const float w = l0 + (l1 - l0) * (float)(p - (ip - 0x1p52));
        v[m] = make_float2(v[m].x * w, v[m].y * w);
    }
    __syncthreads();                                     // every thread has read the forward exchange
    col_fft<N, +1>(v, s, l, t);
    col_store<N>(v, col, es, g.nz, t, c.valid);
}

// ---------------------------------------------------------------- row passes (X)
// Rows are paired two per complex line as in fy_deconv.cuh. TPL neighbouring lanes own a line, so
// a warp transforms 32/TPL lines by itself: the exchange needs no CTA barrier, and rows are read
// and written straight from and to global memory in runs of TPL elements. A line's exchange is
// stored in blocks of PA + 1 points with a line pitch = TPL mod 16 (both conflict-free: a half
// warp's 16/TPL lines fill the banks that one line's TPL lanes leave).
// What bounds them: HBM at 512 (inverse 1.07 GB in 176 us, 0.93 of the measured copy rate;
// 334 us as a shared-memory pass), the L1 data path at the short lengths, whose runs are 4 or 8
// elements wide. Twenty warps an SM at 96 registers: 176 us against 225 us with 24 (spills).
template <int N> struct Row {
    static constexpr int TPL = tpl(N), LPW = 32 / TPL, PA = head_len(N), PB = N / PA;
    static constexpr int pitch0 = PB * (PA + 1);
    static constexpr int pitch = pitch0 + (TPL % 16 + 16 - pitch0 % 16) % 16;
    static constexpr size_t warp_smem = (size_t)LPW * pitch * sizeof(float2), tw_smem = Tail<N>::count * sizeof(float2);
    static constexpr int NT = 128;                        // default threads per CTA
    static constexpr int minb = (elems(N) == 48 ? 16 : (elems(N) == 32 ? 20 : 24)) * 32 / NT;
};
template <int N, int SIGN>
FY_D void row_fft(float2 (&v)[elems(N)], float2* __restrict__ s, int t, const float2* __restrict__ stw) {
    constexpr int PA = head_len(N), Q = PA / tpl(N);
    head<N, SIGN>(v);
    head_store<N>(v, t, [&](int b, int q, float2 x) { s[b * (PA + 1) + q] = x; });
    __syncwarp();
#pragma unroll
    for (int m = 0; m < elems(N); ++m) v[m] = s[(m / Q) * (PA + 1) + t + tpl(N) * (m % Q)];
    tail<N, SIGN>(v, t, stw);
}

// A thread's line: rows 2*line and 2*line + 1 of the nz*ny rows, its lane within the line and the
// half-spectrum rows they fill.
template <int N> struct Line {
    int t;
    long qa;
    long long oa, ob;                                     // spectrum row offsets
    bool ina, inb;
    float2* s;
    FY_D Line(const SpecGeom& g, float2* smem) {
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        t = lane % Row<N>::TPL;
        const int ll = lane / Row<N>::TPL;
        const long line = ((long)blockIdx.x * (blockDim.x >> 5) + w) * Row<N>::LPW + ll;
        const long Q = (long)g.nz * g.ny;
        qa = 2 * line;
        ina = qa < Q;
        inb = qa + 1 < Q;
        const int qi = ina ? (int)qa : 0, z = qi / g.ny, y = qi - z * g.ny;   // nz*ny < 2^31
        oa = ((long long)z * g.py + y) * g.hxp;
        ob = (y + 1 < g.ny ? oa + g.hxp : ((long long)(z + 1) * g.py) * g.hxp);
        s = smem + ((size_t)w * Row<N>::LPW + ll) * Row<N>::pitch;
    }
};

// X forward: rows (u8 dewindowed, or f32), reflect padding, transform, untangle, half spectra.
// The mirrored point N - k of the untangle sits in lane TPL - t (lane 0: its own), one shuffle.
template <int N, class T, bool PAD>
__global__ void __launch_bounds__(Row<N>::NT, Row<N>::minb)
k_row_fwd(const T* __restrict__ src, float lo, float scale, float2* __restrict__ spec, SpecGeom g,
          const float2* __restrict__ tw) {
    fy_pdl_wait();
    extern __shared__ float4 smem4[];
    constexpr int E = elems(N), TPL = tpl(N);
    float2* stw = reinterpret_cast<float2*>(smem4);
    const Line<N> ln(g, stw + Tail<N>::count);
    const int t = ln.t;
    const T* pa = src + (ln.ina ? ln.qa : 0) * g.nx;
    const T* pb = ln.inb ? pa + g.nx : pa;
    float2 v[E];
#pragma unroll
    for (int m = 0; m < E; ++m) {
        const int i = t + TPL * m, x = PAD ? pad_src(i, g.nx) : i;
        float a = (float)__ldg(pa + x), b = (float)__ldg(pb + x);
        if (sizeof(T) == 1) {                             // fy_u8_to_phys, FMA as the reference build
            a = __fmaf_rn(a, scale, lo);
            b = __fmaf_rn(b, scale, lo);
        }
        v[m] = make_float2(ln.ina ? a : 0.f, ln.inb ? b : 0.f);
    }
    load_tail_twiddles<N>(stw, tw);
    __syncthreads();
    row_fft<N, -1>(v, ln.s, t, stw);
    const int mlane = (threadIdx.x & 31) - t + (TPL - t) % TPL;
    float2* sa = spec + ln.oa;
    float2* sb = spec + ln.ob;
#pragma unroll
    for (int m = 0; m < E / 2; ++m) {
        const float2 own = v[(E - m) % E], oth = v[E - 1 - m];
        float2 M = t == 0 ? own : oth, A, B;
        if (TPL > 1) {
            M.x = __shfl_sync(0xffffffffu, M.x, mlane);
            M.y = __shfl_sync(0xffffffffu, M.y, mlane);
        }
        untangle(v[m], M, A, B);
        if (ln.ina) sa[t + TPL * m] = A;
        if (ln.inb) sb[t + TPL * m] = B;
    }
    if (t == 0) {                                         // k = N/2 is its own mirror
        float2 A, B;
        untangle(v[E / 2], v[E / 2], A, B);
        if (ln.ina) sa[N / 2] = A;
        if (ln.inb) sb[N / 2] = B;
    }
}

// X inverse: the two half spectra of a line, pack (mirrored points by the same shuffle), inverse
// transform, crop, 1/N.
template <int N, bool CROP>
__global__ void __launch_bounds__(Row<N>::NT, Row<N>::minb)
k_row_inv(const float2* __restrict__ spec, float* __restrict__ dst, int dpitch, SpecGeom g, const float2* __restrict__ tw, float invN) {
    fy_pdl_wait();
    extern __shared__ float4 smem4[];
    constexpr int E = elems(N), TPL = tpl(N), H = E / 2;
    float2* stw = reinterpret_cast<float2*>(smem4);
    const Line<N> ln(g, stw + Tail<N>::count);
    const int t = ln.t, mlane = (threadIdx.x & 31) - t + (TPL - t) % TPL;
    const float2 zero = make_float2(0.f, 0.f);
    const float2* sa = spec + (ln.ina ? ln.oa : 0);
    const float2* sb = spec + (ln.inb ? ln.ob : 0);
    float2 v[E];
#pragma unroll
    for (int m = 0; m < H; ++m) {
        v[m] = ln.ina ? __ldg(sa + t + TPL * m) : zero;
        v[H + m] = ln.inb ? __ldg(sb + t + TPL * m) : zero;
    }
    float2 nyq = zero;
    if (t == 0) nyq = pack_lo(ln.ina ? __ldg(sa + N / 2) : zero, ln.inb ? __ldg(sb + N / 2) : zero);
    // v[m] := lo_m and v[E-1-m] := the mirrored hi of lane TPL - t, pair by pair (the pair's two
    // B slots are the two slots it fills)
#pragma unroll
    for (int m = 0; m < H / 2; ++m) {
        const int n = H - 1 - m;
        const float2 A0 = v[m], B0 = v[H + m], A1 = v[n], B1 = v[H + n];
        v[m] = pack_lo(A0, B0);
        v[n] = pack_lo(A1, B1);
        float2 h0 = pack_hi(A0, B0), h1 = pack_hi(A1, B1);
        if (TPL > 1) {
            h0.x = __shfl_sync(0xffffffffu, h0.x, mlane);
            h0.y = __shfl_sync(0xffffffffu, h0.y, mlane);
            h1.x = __shfl_sync(0xffffffffu, h1.x, mlane);
            h1.y = __shfl_sync(0xffffffffu, h1.y, mlane);
        }
        v[E - 1 - m] = h0;
        v[E - 1 - n] = h1;
    }
    // lane 0's mirrors sit one slot higher (N - k = TPL*(E - m)), and slot E/2 is k = N/2
#pragma unroll
    for (int i = E - 1; i > H; --i) v[i] = t == 0 ? v[i - 1] : v[i];
    v[H] = t == 0 ? nyq : v[H];
    load_tail_twiddles<N>(stw, tw);
    __syncthreads();
    row_fft<N, +1>(v, ln.s, t, stw);
    float* da = dst + ln.qa * dpitch;
    float* db = da + dpitch;
#pragma unroll
    for (int m = 0; m < E; ++m) {
        const int x = t + TPL * m;
        if (CROP && x >= g.nx) continue;
        if (ln.ina) da[x] = v[m].x * invN;
        if (ln.inb) db[x] = v[m].y * invN;
    }
}

// Threads per CTA of a row pass: NT, halved once for each power of two that a tuned lines-per-CTA
// value lies below the shared-memory tile's (fy_x_tile_shape), never below a warp.
template <int N>
inline int row_threads(int pass) {
    const int d = fy_tile_shape(N).wlog - fy_x_tile_shape(pass, N).wlog;
    const int nt = Row<N>::NT >> (d > 0 ? d : 0);
    return nt < 32 ? 32 : nt;
}

template <class K, class... A>
inline cudaError_t launch(K k, unsigned grid, int nt, size_t smem, cudaStream_t st, A... a) {
    const cudaError_t e = fy_smem_optin(k, smem);
    return e != cudaSuccess ? e : fy_launch_pdl(k, dim3(grid), dim3(nt), smem, st, a...);
}

// A Y pass over `nplanes` stored planes; sign -1: rows >= ny gathered by reflection, every row
// stored; sign +1: rows < keep_rows stored.
template <int N>
inline cudaError_t launch_y(float2* spec, const SpecGeom& g, const float2* tw, int nplanes, int sign, int keep_rows,
                            int sms, cudaStream_t st) {
    using C = Col<N>;
    const ColTiles ct = col_tiles(g.hx, nplanes, C::W, N <= 256 ? 2L * sms * C::minb : LONG_MAX);
    if (sign > 0) return launch(k_col_y<N, 1, false>, ct.total, C::NT, C::smem, st, spec, g, ct, tw, N, keep_rows);
    if (g.ny == N) return launch(k_col_y<N, -1, false>, ct.total, C::NT, C::smem, st, spec, g, ct, tw, N, N);
    return launch(k_col_y<N, -1, true>, ct.total, C::NT, C::smem, st, spec, g, ct, tw, g.ny, N);
}

// Pass `pass` (1..5) of a deconvolution whose axis length there is N.
template <int N>
cudaError_t deconv_pass(int pass, const DeconvLaunch& d, cudaStream_t st) {
    const SpecGeom& g = d.g;
    const long lines = ((long)g.nz * g.ny + 1) / 2;
    auto rows = [&](int nt) { const long per = (long)(nt / 32) * Row<N>::LPW; return (unsigned)((lines + per - 1) / per); };
    switch (pass) {
    case 1: {
        const int nt = row_threads<N>(1);
        const size_t smem = Row<N>::tw_smem + Row<N>::warp_smem * (nt / 32);
        const bool pad = g.nx != N;
#define FY_ROW_FWD(T, P) launch(k_row_fwd<N, T, P>, rows(nt), nt, smem, st, (const T*)d.src, d.lo, d.scale, d.spec, g, d.twx)
        if (d.src_u8) return pad ? FY_ROW_FWD(uint8_t, true) : FY_ROW_FWD(uint8_t, false);
        return pad ? FY_ROW_FWD(float, true) : FY_ROW_FWD(float, false);
#undef FY_ROW_FWD
    }
    case 2: return launch_y<N>(d.spec, g, d.twy, g.nz, -1, g.py, d.sms, st);
    case 4: return launch_y<N>(d.spec, g, d.twy, g.nz, +1, g.ny, d.sms, st);
    case 3: {
        using C = Col<N>;
        const ColTiles ct = col_tiles(g.hx, g.py, C::W, (long)d.sms * C::minb);
        if (g.nz == N)
            return launch(k_col_z<N, false>, ct.total, C::NT, C::smem, st, d.spec, g, ct, d.twz, d.lut, d.fz2, d.fy2, d.fx2, d.us);
        return launch(k_col_z<N, true>, ct.total, C::NT, C::smem, st, d.spec, g, ct, d.twz, d.lut, d.fz2, d.fy2, d.fx2, d.us);
    }
    case 5: {
        const int nt = row_threads<N>(5);
        const size_t smem = Row<N>::tw_smem + Row<N>::warp_smem * (nt / 32);
        const float invN = 1.0f / ((float)g.pz * (float)g.py * (float)g.px);   // paganin.c:263
        if (g.nx != N) return launch(k_row_inv<N, true>, rows(nt), nt, smem, st, (const float2*)d.spec, d.dst, d.dpitch, g, d.twx, invN);
        return launch(k_row_inv<N, false>, rows(nt), nt, smem, st, (const float2*)d.spec, d.dst, d.dpitch, g, d.twx, invN);
    }
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace rf
