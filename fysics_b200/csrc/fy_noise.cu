// fy_noise.cu -- per-volume noise model fy_estimate_noise (noise.c:75-192) on the GPU.
//
//   1. Local stats, a z-sliding box pass (fy_zbox.cuh): box sums over (2r+1)^3 windows with
//      zero outside the volume and the FIXED divisor win^3 (noise.c:20-59, 92-101): mean m
//      and variance v = max(S2/wc - m^2, 0). Sums are direct
//      (2r+1)-tap float sums of (I - c) and (I - c)^2 with a per-tile shift c, and interior
//      voxels use v = S2'/wc - (S1'/wc)^2, which equals the reference's S2/wc - (S1/wc)^2
//      without its cancellation.
//   2. Exact order statistics on orderable 32-bit float keys: the 1st and 99th percentiles
//      of m (noise.c:104-108) and, per intensity bin with >= 200 voxels, the flat_pct percentile
//      of v (noise.c:117-134), each interpolated between order statistics k and k+1 exactly as
//      percentile() does (noise.c:66-73). Each of the two selections reads its fields once, through
//      sample-guided windows (section 2w): sample and bounds, count, bucket, collect. Radix passes
//      over the window's candidates or over the whole field stand behind them (section 2r) and
//      exit at once when the windows gave the answer.
//   3. k_noise_fit: one warp, FP64 (five lanes form the weighted sums): IRLS line fit
//      var = g*I + b (noise.c:137-172) and noise_ref = sqrt(max(g*ref + b, ..))*1.15 (noise.c:181-187), plus the guided eps
//      (3*noise_ref)^2 floored at 1e-8 (noise.c:197-202).
// The launch sequence is fixed (no host decisions), so a chain can keep it on one stream.
#include <cuda/std/tuple>
#include <vector>

#include "fy_internal.h"
#include "fysics_b200.h"
#include "fy_zbox.cuh"

namespace {

constexpr int NB = 24;                 // intensity bins, noise.c:111
// ctl->mode: which step acts next. The window steps of the means (kMeanWin) and of the bins
// (kBinWin) hand over to their radix passes: over the candidates (kMeanCand, kBinCand) when one
// bucket holds too many keys to collect, over the whole field (kMeanField, kBinField) when a
// window missed or its candidate list overflowed. kVarField: no bin qualifies, the percentile of
// all variances (noise.c:166-171).
enum { kMeanWin, kMeanCand, kMeanField, kBinWin, kBinCand, kBinField, kVarField };

FY_D uint32_t fkey(float f) {
    const uint32_t u = __float_as_uint(f);
    return u ^ ((uint32_t)((int32_t)u >> 31) | 0x80000000u);   // negative: ~u, else u | sign
}
FY_HD float funkey(uint32_t k) {
#ifdef __CUDA_ARCH__
    const uint32_t u = (k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k;
    return __uint_as_float(u);
#else
    const uint32_t u = (k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k;
    float f;
    memcpy(&f, &u, 4);
    return f;
#endif
}

}  // namespace

// Device-resident control block of one estimate (lives in the caller's scratch).
// Selection targets: target t selects the order statistic k_t (0-based) of the keys of its
// group: the 1st/99th percentile (t = 0, 1), a bin (t = bin), or all variances (t = 0). When a
// selection has ended, prefix_t is the k-th key, and the (k+1)-th is the same key unless
// tneed_next, then tnext.
constexpr int kHist = NB * 256;        // the targets' histograms: 256 digits each, or window buckets
struct NoiseCtl {
    long long n;
    double flat_pct, ref_intensity;
    int ntarget, mode;
    long long tk[NB];                  // requested rank k
    long long trank[NB];               // remaining rank inside the decided prefix
    long long tgroup_n[NB];            // group size
    unsigned long long teq[NB];        // keys equal to the selected key
    uint32_t tprefix[NB];
    uint32_t tnext[NB];                // smallest key above the selected one (when needed)
    uint32_t tabove[NB];               // radix passes: smallest key above the last digit's prefix
    int tactive[NB];
    int tneed_next[NB];
    double edge[NB + 1];
    float fedge[NB + 1];               // smallest float >= edge[k]: exact float membership test
    unsigned long long bcount[NB];
    double out_g, out_b, out_noise_ref, out_ref_intensity;
    int out_used;
    float eps;                         // fy_guided_eps_for_noise(noise_ref), for a chained guided filter
    alignas(16) unsigned int hist[kHist];
    // windows (section 2w): per target the keys [wlo, whi], the group's keys below wlo and, for a
    // bin, its voxels; the candidate list's length; the bucket origin and scale of the window's
    // values; the buckets that hold the ranks k and k+1, the rank within them and the keys collected
    uint32_t wlo[NB], whi[NB];
    uint32_t klo[NB], khi[NB];         // the sample's keys that bound the window (its ends, where it has some)
    unsigned long long wbelow[NB], wvox[NB];
    unsigned long long ncand;          // candidates appended (may exceed the capacity)
    float cv0[NB], cvs[NB];
    int cb0[NB], cb1[NB];
    long long crank[NB];
    unsigned int ccnt[NB];
    unsigned int bsn[NB];              // sample keys listed per bin (may exceed the list's capacity)
    unsigned int done_ctas;            // CTAs of the current step that have finished (0 between steps)
};

namespace {


// The block index and grid size along x of the CTA's volume, which every selection body uses
// in place of blockIdx.x / gridDim.x: k_one sets them from its launch, k_many from the step's
// table of CTAs per volume (a batch launch holds every volume's CTAs along x).
static __shared__ unsigned s_vbx, s_vgx;
FY_D unsigned vbx() { return s_vbx; }
FY_D unsigned vgx() { return s_vgx; }

// ---------------------------------------------------------------- 1. local stats
// z-sliding box pass (fy_zbox.cuh, ZB_NOISE): 4 B read + 8 B written per voxel.

// The CTA of the volume that gets here last (a ticket) returns true, with every other CTA's
// writes before its own ticket visible; it then sets done_ctas back to 0.
FY_D bool last_cta(NoiseCtl* ctl) {
    __shared__ int s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&ctl->done_ctas, 1u) == vgx() - 1;
    __syncthreads();
    if (!s_last) return false;
    __threadfence();
    return true;
}

FY_D void target_init(NoiseCtl* ctl, int t, long long k, long long group_n, bool on) {
    ctl->tk[t] = k;
    ctl->trank[t] = k;
    ctl->tgroup_n[t] = group_n;
    ctl->tprefix[t] = 0;
    ctl->teq[t] = 0;
    ctl->tactive[t] = on;
    ctl->tneed_next[t] = 0;
    ctl->tnext[t] = 0xffffffffu;
    ctl->tabove[t] = 0xffffffffu;
}

// ---------------------------------------------------------------- 2r. radix select
// Exact bin of a float mean: m >= edge[k] <=> m >= fedge[k] with fedge[k] the smallest float
// >= edge[k] (noise.c:118-122 in double), so membership needs only float compares.
FY_D int bin_of(float m, const float* __restrict__ fe, float lo_f, float scale) {
    if (!(m >= fe[0] && m < fe[NB])) return -1;
    int b = (int)((m - lo_f) * scale);
    b = b < 0 ? 0 : (b > NB - 1 ? NB - 1 : b);
    while (b > 0 && m < fe[b]) --b;
    while (b < NB - 1 && m >= fe[b + 1]) ++b;
    return b;
}

// Histogram increments with thread-local run merging: a thread's consecutive equal codes
// are counted in a register and added with one shared atomic per run. Neighbouring voxels
// mostly share intensity bins and high digits, so concentrated passes make few atomics,
// and spread-out passes pay only bank conflicts; no warp collectives are needed.
struct RunAcc {
    int cur = -1;
    unsigned int cnt = 0;
    FY_D void add(unsigned int* h, int code) {
        if (code != cur) {
            if (cur >= 0) atomicAdd(&h[cur], cnt);
            cur = code;
            cnt = 0;
        }
        ++cnt;
    }
    FY_D void flush(unsigned int* h) {
        if (cur >= 0) atomicAdd(&h[cur], cnt);
        cur = -1;
        cnt = 0;
    }
};

struct WarpCands {
    float* v;                          // this warp's values in shared memory
    uint8_t* l;                        // and labels
    int cnt = 0;                       // warp-uniform fill
    FY_D void flush(float* __restrict__ cval, uint8_t* __restrict__ clab, unsigned long long* ncand, long long cap) {
        const unsigned full = 0xffffffffu;
        __syncwarp();
        if (cnt) {
            unsigned long long base = 0;
            if ((threadIdx.x & 31) == 0) base = atomicAdd(ncand, (unsigned long long)cnt);
            base = __shfl_sync(full, base, 0);
            for (int i = threadIdx.x & 31; i < cnt; i += 32)
                if ((long long)(base + i) < cap) { cval[base + i] = v[i]; clab[base + i] = l[i]; }
        }
        cnt = 0;
        __syncwarp();
    }
};

// Streaming passes read SU float4 (and uchar4 bin labels) per thread before using any, so
// enough bytes are in flight per SM to cover HBM latency. Full chunks of the grid-stride
// loop run without per-element range checks; the one partial chunk is checked.
constexpr int SU = 4;

// The bookkeeping after a digit pass for target t, by one warp: the bucket that holds the
// target's rank (a warp scan of the lanes' bucket sums), the prefix extended by it, the keys
// equal to the selected key and, after the last digit, the smallest key above the selected one:
// the next non-empty bucket within the prefix, else the smallest key above the prefix, which
// the last pass recorded. The histogram is read through L2 (other CTAs' atomics) and cleared.
FY_D void warp_scan_target(NoiseCtl* ctl, int t, bool last) {
    constexpr int per = 256 / 32;
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    unsigned int* h = ctl->hist + t * 256;
    const int b0 = lane * per;
    const long long r = ctl->trank[t];
    const uint32_t pre = ctl->tprefix[t];
    unsigned int hv[per];
    unsigned long long mine = 0;
#pragma unroll
    for (int i = 0; i < per; ++i) hv[i] = __ldcg(h + b0 + i);
#pragma unroll
    for (int i = 0; i < per; ++i) mine += hv[i];
    unsigned long long incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(full, incl, o);
        if (lane >= o) incl += y;
    }
    const unsigned long long before = incl - mine;
    unsigned int sel = 256;
    if ((unsigned long long)r >= before && (unsigned long long)r < incl) {
        unsigned long long acc = before;
        unsigned int hsel = 0;
#pragma unroll
        for (int i = 0; i < per; ++i) {
            if (sel == 256 && acc + hv[i] > (unsigned long long)r) { sel = (unsigned)(b0 + i); hsel = hv[i]; }
            else if (sel == 256) acc += hv[i];
        }
        ctl->trank[t] = r - (long long)acc;
        ctl->tprefix[t] = (pre << 8) | sel;
        if (last) ctl->teq[t] = hsel;
    }
    sel = __reduce_min_sync(full, sel);
    unsigned int nextb = 0xffffffffu;
    if (last) {
#pragma unroll
        for (int i = per - 1; i >= 0; --i)
            if (b0 + i > (int)sel && hv[i]) nextb = (unsigned)(b0 + i);
        nextb = __reduce_min_sync(full, nextb);
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < per; ++i) h[b0 + i] = 0;
    __syncwarp();
    if (last && lane == 0) {
        ctl->tneed_next[t] = (ctl->trank[t] + 1 >= (long long)ctl->teq[t]) && (ctl->tk[t] + 1 < ctl->tgroup_n[t]);
        ctl->tnext[t] = nextb != 0xffffffffu ? (pre << 8) | nextb : __ldcg(&ctl->tabove[t]);
    }
}

// One 8-bit digit pass (bits [shift, shift + 8)) over n keys for every active target whose prefix
// matches. LAB 0: no labels, every key belongs to every target (at most two; targets whose
// prefixes are equal share one shared-memory histogram, so a key makes at most one increment, and
// the flush copies a group's counts to each of its targets). LAB 1: the key's target is its u8
// label. LAB 2 (the first pass over the bins): the label is computed from the voxel's mean and
// written for the later passes. Inactive targets and label 255 carry the prefix 0xffffffff, which
// no key's high part can equal. The last pass also records, per target, the smallest key above
// the prefix.
template <int LAB>
FY_D void radix_pass(const float* __restrict__ src, const float* __restrict__ mean, uint8_t* __restrict__ lab8,
                     long long n, NoiseCtl* __restrict__ ctl, int shift, unsigned int* __restrict__ h) {
    __shared__ uint32_t sp[256];
    __shared__ unsigned int smin[NB];
    __shared__ float fe[NB + 1];
    const int nt = ctl->ntarget, top = shift + 8;
    if (LAB == 2 && threadIdx.x <= NB) fe[threadIdx.x] = ctl->fedge[threadIdx.x];
    for (int i = threadIdx.x; i < 256; i += blockDim.x) sp[i] = i < nt && ctl->tactive[i] ? ctl->tprefix[i] : 0xffffffffu;
    if (threadIdx.x < NB) smin[threadIdx.x] = 0xffffffffu;
    uint32_t p0 = 0xffffffffu, p1 = 0xffffffffu;
    int g1 = 1;                                          // target 1's histogram: 0 when it shares target 0's prefix
    if (LAB == 0) {
        if (ctl->tactive[0]) p0 = ctl->tprefix[0];
        if (nt > 1 && ctl->tactive[1]) {
            p1 = ctl->tprefix[1];
            if (p1 == p0) { g1 = 0; p1 = 0xfffffffeu; }  // never matches
        }
    }
    for (int i = threadIdx.x; i < (LAB == 0 ? 2 : nt) * 256; i += blockDim.x) h[i] = 0;
    __syncthreads();
    const float lo_f = LAB == 2 ? fe[0] : 0.f, fscale = LAB == 2 ? (float)(NB / (ctl->edge[NB] - ctl->edge[0])) : 0.f;
    auto label = [&](float m) -> unsigned { const int b = bin_of(m, fe, lo_f, fscale); return b < 0 ? 255u : (unsigned)b; };
    RunAcc acc;
    uint32_t a0 = 0xffffffffu, a1 = 0xffffffffu;          // LAB 0: smallest key above the prefix of targets 0, 1
    const uint32_t q1 = g1 ? p1 : p0;
    auto visit = [&](float v, unsigned g) {
        const uint32_t key = fkey(v);
        const uint32_t hb = top >= 32 ? 0u : (key >> top);
        const int dig = (key >> shift) & 255;
        if (LAB) {
            const uint32_t pg = sp[g];
            acc.add(h, pg == hb ? (int)g * 256 + dig : -1);
            if (shift == 0 && hb > pg && key < smin[g]) atomicMin(&smin[g], key);
        } else {
            acc.add(h, hb == p0 ? dig : (hb == p1 ? 256 + dig : -1));
            if (shift == 0) {
                if (hb > p0) a0 = min(a0, key);
                if (hb > q1) a1 = min(a1, key);
            }
        }
    };
    const int step = blockDim.x;
    const long long n4 = (n + 3) / 4, n4f = n / 4, chunk = (long long)SU * step;
    long long base = (long long)vbx() * chunk;
    const long long stride = (long long)vgx() * chunk;        // read once: the loop body has syncs
    for (; base + chunk <= n4f; base += stride) {
        float4 x[SU];
        uchar4 bb[SU];
        float4 mm[LAB == 2 ? SU : 1];
#pragma unroll
        for (int u = 0; u < SU; ++u) {
            const long long q = base + threadIdx.x + (long long)u * step;
            x[u] = __ldg(reinterpret_cast<const float4*>(src) + q);
            if (LAB == 2) mm[u] = __ldg(reinterpret_cast<const float4*>(mean) + q);
            else if (LAB) bb[u] = *(reinterpret_cast<const uchar4*>(lab8) + q);
        }
#pragma unroll
        for (int u = 0; u < SU; ++u) {
            if (LAB == 2) {
                bb[u] = make_uchar4(label(mm[u].x), label(mm[u].y), label(mm[u].z), label(mm[u].w));
                reinterpret_cast<uchar4*>(lab8)[base + threadIdx.x + (long long)u * step] = bb[u];
            }
            visit(x[u].x, LAB ? bb[u].x : 0);
            visit(x[u].y, LAB ? bb[u].y : 0);
            visit(x[u].z, LAB ? bb[u].z : 0);
            visit(x[u].w, LAB ? bb[u].w : 0);
        }
    }
    if (base < n4) {                                     // the grid's partial chunk
        for (int u = 0; u < SU; ++u)
            for (int j = 0; j < 4; ++j) {
                const long long i = 4 * (base + threadIdx.x + (long long)u * step) + j;
                if (i >= n) continue;
                unsigned g = 0;
                if (LAB == 2) { g = label(__ldg(mean + i)); lab8[i] = (uint8_t)g; }
                else if (LAB) g = lab8[i];
                visit(__ldg(src + i), g);
            }
    }
    acc.flush(h);
    if (LAB == 0 && shift == 0) {
        if (a0 != 0xffffffffu) atomicMin(&smin[0], a0);
        if (a1 != 0xffffffffu) atomicMin(&smin[1], a1);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nt * 256; i += blockDim.x) {
        const int t = i >> 8;
        const unsigned int cnt = h[LAB ? i : (t == 0 ? 0 : g1) * 256 + (i & 255)];
        if (cnt) atomicAdd(&ctl->hist[i], cnt);
    }
    if (shift == 0 && threadIdx.x < nt && smin[threadIdx.x] != 0xffffffffu)
        atomicMin(&ctl->tabove[threadIdx.x], smin[threadIdx.x]);
    if (!last_cta(ctl)) return;
    for (int t = threadIdx.x >> 5; t < nt; t += blockDim.x >> 5)
        if (ctl->tactive[t]) warp_scan_target(ctl, t, shift == 0);
    if (threadIdx.x == 0) ctl->done_ctas = 0;
}

// The radix passes behind the means' windows, and behind the bins': which keys a pass reads
// follows from ctl->mode; in the common case none, and the launch ends at once.
FY_D void k_mean_radix(const float* __restrict__ mean, NoiseCtl* __restrict__ ctl, const float* __restrict__ cval,
                       uint8_t* __restrict__ clab, int shift) {
    fy_pdl_wait();
    extern __shared__ unsigned int rh[];
    const int mode = ctl->mode;
    if (mode == kMeanField) radix_pass<0>(mean, nullptr, nullptr, ctl->n, ctl, shift, rh);
    else if (mode == kMeanCand) radix_pass<1>(cval, nullptr, clab, (long long)ctl->ncand, ctl, shift, rh);
}
FY_D void k_bin_radix(const float* __restrict__ mean, const float* __restrict__ var, uint8_t* __restrict__ bin,
                      NoiseCtl* __restrict__ ctl, const float* __restrict__ cval, uint8_t* __restrict__ clab, int shift) {
    fy_pdl_wait();
    extern __shared__ unsigned int rh[];
    const int mode = ctl->mode;
    if (mode == kBinField) {
        if (shift == 24) radix_pass<2>(var, mean, bin, ctl->n, ctl, shift, rh);
        else radix_pass<1>(var, nullptr, bin, ctl->n, ctl, shift, rh);
    } else if (mode == kBinCand) radix_pass<1>(cval, nullptr, clab, (long long)ctl->ncand, ctl, shift, rh);
    else if (mode == kVarField) radix_pass<0>(var, nullptr, nullptr, ctl->n, ctl, shift, rh);
}

// value of order statistic k+1 of target t
FY_D double next_value(const NoiseCtl* ctl, int t) {
    return ctl->tneed_next[t] ? (double)funkey(ctl->tnext[t]) : (double)funkey(ctl->tprefix[t]);
}
// percentile() interpolation (noise.c:69-72)
FY_D double interp(const NoiseCtl* ctl, int t, double f, bool has_next) {
    const double v0 = (double)funkey(ctl->tprefix[t]);
    if (!has_next) return v0;
    return v0 * (1 - f) + next_value(ctl, t) * f;
}

// ---------------------------------------------------------------- 2w. sample-guided windows
// A selection by radix passes alone reads its field once per digit. Here it reads it once:
//   sample   values at positions (A*i + B) mod n, a bijection of [0, n) when gcd(A, n) = 1,
//            spread evenly over the volume: 16384 means; 65536 (mean, variance) pairs, listed per
//            intensity bin.
//   bounds   per target the sample's order statistics kWinSigmas binomial standard deviations
//            either side of its expected sample rank give a key window [wlo, whi] that holds the
//            order statistics k and k+1 with overwhelming probability (block_bounds).
//   count    one pass over the field(s) counts, per target, the keys below wlo and appends the
//            keys inside to a candidate list with their target; for the bins it also gives the
//            bin counts, which set k.
//   bucket   the candidates' histogram over equal steps of value in the window (a step's bucket
//            is a monotone function of the key, so buckets are in key order): the bucket of the
//            rank r = k - below, and of r + 1.
//   collect  the keys of those buckets (a few hundred; up to kListMax) into a list per target.
//   select   one CTA per target selects among them in registers.
// Every step's closing bookkeeping runs in its last CTA. A rank outside its
// window or a candidate list over its capacity sends the selection to the radix passes over the
// whole field; buckets with too many keys to collect (ties) send it to the radix passes over the
// candidates. All of them give the same exact order statistics.
constexpr int kSampleMax = 16384;
constexpr int kBinSampleMax = 65536;
constexpr int kBinListMax = 16384;     // sample keys per bin: a window of 2.4% of the largest bins
constexpr int kBinListSmall = 2048;    // in the scratch's own region, for fields of few candidates
constexpr int kListMax = 16384;        // keys that a target can collect
constexpr int kBoundThreads = 1024;    // CTAs that select among keys in registers
constexpr int kKeysPerThread = 16;
static_assert(kSampleMax <= kBoundThreads * kKeysPerThread && kBinListMax <= kBoundThreads * kKeysPerThread &&
              kListMax <= kBoundThreads * kKeysPerThread, "every list fits the block's registers");
constexpr double kWinSigmas = 5.0;
// Test hook: bit 0 forces the mean percentiles, bit 1 the bins, to the radix passes over the
// whole field, bits 2 and 3 to those over the windows' candidates; noise_window_used records (bits
// 0/1) which windows produced their result and (bits 2/3) which of them by the candidates' passes.
static __device__ int noise_force_radix;
static __device__ int noise_window_used;

// The bucket that holds rank r in a shared-memory histogram of nh buckets (a power of two, 64 to
// 2048), and the keys before it; by one warp (every lane gets them; r is below the total). The lanes
// sum nh/32 buckets each (read rotated: few bank conflicts), then share the rank's segment.
FY_D void warp_find(const unsigned int* __restrict__ h, int nh, unsigned int r, int& bucket, unsigned int& before) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, per = nh >> 5;
    auto scan = [&](unsigned int v) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned int y = __shfl_up_sync(full, v, o);
            if (lane >= o) v += y;
        }
        return v;
    };
    unsigned int sum = 0;
#pragma unroll 8
    for (int i = 0; i < per; ++i) sum += h[lane * per + ((i + lane) & (per - 1))];
    unsigned int incl = scan(sum);
    const int seg = __ffs(__ballot_sync(full, r < incl)) - 1;
    const unsigned int base = __shfl_sync(full, incl - sum, seg);
    const unsigned int* hs = h + seg * per;               // at most 64 buckets: two per lane
    const unsigned int v0 = 2 * lane < per ? hs[2 * lane] : 0u, v1 = 2 * lane + 1 < per ? hs[2 * lane + 1] : 0u;
    incl = scan(v0 + v1);
    const int l = __ffs(__ballot_sync(full, r - base < incl)) - 1;
    unsigned int acc = base + incl - v0 - v1;
    int b = seg * per + 2 * lane;
    if (acc + v0 <= r) { acc += v0; ++b; }
    bucket = __shfl_sync(full, b, l);
    before = __shfl_sync(full, acc, l);
}

// NQ order statistics of the CTA's keys (kKeysPerThread per thread in registers, thread t's i-th is
// number t + i*kBoundThreads, c >= 1 of them valid; ranks 0-based < c). Histograms of 2048 equal key
// steps over the keys' range, then inside each rank's bucket: lo <= statistic <= hi, hi - lo below
// 2^-22 of the range. EXACT: and inside that, lo = statistic. sh: (NQ + 1) * 2048 counters.
template <int NQ, bool EXACT>
FY_D void block_stats(const uint32_t (&k)[kKeysPerThread], int c, const int (&rank)[NQ], unsigned int* __restrict__ sh,
                      uint32_t (&lo)[NQ], uint32_t (&hi)[NQ]) {
    constexpr int NH = 2048, NTB = kBoundThreads, KPT = kKeysPerThread;
    __shared__ uint32_t s_min, s_max;
    __shared__ unsigned int s_b[NQ], s_r[NQ];
    const unsigned full = 0xffffffffu;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    if (t == 0) { s_min = 0xffffffffu; s_max = 0u; }
    for (int i = t; i < (NQ + 1) * NH; i += NTB) sh[i] = 0;
    __syncthreads();
    uint32_t mn = 0xffffffffu, mx = 0u;
#pragma unroll
    for (int i = 0; i < KPT; ++i)
        if (t + i * NTB < c) { mn = min(mn, k[i]); mx = max(mx, k[i]); }
    mn = __reduce_min_sync(full, mn);
    mx = __reduce_max_sync(full, mx);
    if (lane == 0 && mn <= mx) { atomicMin(&s_min, mn); atomicMax(&s_max, mx); }
    __syncthreads();
    const uint32_t k0 = s_min, range = s_max - k0;
    const int bits = 32 - __clz(range), sh1 = bits > 11 ? bits - 11 : 0, sh2 = sh1 > 11 ? sh1 - 11 : 0;
#pragma unroll
    for (int i = 0; i < KPT; ++i)
        if (t + i * NTB < c) atomicAdd(&sh[(k[i] - k0) >> sh1], 1u);
    __syncthreads();
    auto find = [&](const unsigned int* h, unsigned int r) {    // warp q < NQ
        int b;
        unsigned int before;
        warp_find(h, NH, r, b, before);
        if (lane == 0) {
            s_b[w] = (unsigned)b;
            s_r[w] = r - before;
        }
    };
    if (w < NQ) find(sh, (unsigned)rank[w]);
    __syncthreads();
    uint32_t pre[NQ];                                    // (key - k0) >> the level's shift, per rank
#pragma unroll
    for (int q = 0; q < NQ; ++q) pre[q] = s_b[q];
    auto level = [&](int from, int to) {                 // refine the buckets of shift `from` to shift `to`
#pragma unroll
        for (int i = 0; i < KPT; ++i) {
            if (t + i * NTB >= c) continue;
            const uint32_t d = k[i] - k0, b = d >> from, sub = (d & ((1u << from) - 1u)) >> to;
#pragma unroll
            for (int q = 0; q < NQ; ++q)
                if (b == pre[q]) atomicAdd(&sh[(q + 1) * NH + sub], 1u);
        }
        const unsigned int r = w < NQ ? s_r[w] : 0u;
        __syncthreads();
        if (w < NQ) find(sh + (w + 1) * NH, r);
        __syncthreads();
#pragma unroll
        for (int q = 0; q < NQ; ++q) pre[q] = (pre[q] << (from - to)) + s_b[q];
    };
    if (sh1 > 0) level(sh1, sh2);
    if (EXACT && sh2 > 0) {
        for (int i = t; i < NQ * NH; i += NTB) sh[NH + i] = 0;
        __syncthreads();
        level(sh2, 0);
    }
    const int last = EXACT ? 0 : sh2;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        lo[q] = k0 + (pre[q] << last);
        hi[q] = lo[q] + ((1u << last) - 1u);
    }
}

// The sample ranks either side of quantile q of c samples (lo < 0 or hi >= c: none).
FY_D void window_ranks(double q, int c, int& lo, int& hi) {
    const double qc = q < 1.0 / c ? 1.0 / c : (q > 1.0 - 1.0 / c ? 1.0 - 1.0 / c : q);
    const int ks = (int)(q * (double)(c - 1));
    const int d = (int)ceil(kWinSigmas * sqrt((double)c * qc * (1.0 - qc))) + 4;
    lo = ks - d;
    hi = ks + d + 1;
}

// Value buckets of a window: origin and scale of nb equal steps between the sample's keys that
// bound it (an open window ends at the sample's extremes, so that the bulk of its keys is spread;
// keys beyond fall into the end buckets). Whatever they are, bucket_of is monotone in the key.
FY_D void window_buckets(NoiseCtl* ctl, int t, int nb) {
    const uint32_t kmin = 0x00800000u, kmax = 0xff7fffffu;          // keys of -FLT_MAX and FLT_MAX
    const uint32_t a = min(max(ctl->klo[t], kmin), kmax), b = min(max(ctl->khi[t], kmin), kmax);
    const float v0 = funkey(a), d = funkey(b) - v0;
    ctl->cv0[t] = v0;
    ctl->cvs[t] = d > 0.f ? (float)nb / d : 0.f;
}
FY_D int bucket_of(float v, float v0, float s, int nb) {
    const int b = (int)((v - v0) * s);                               // saturates; NaN gives 0
    return fkey(v) > 0xff800000u ? nb - 1 : min(max(b, 0), nb - 1);  // positive NaNs are the largest keys
}

// One CTA per volume: the control block, and the windows of the 1st/99th percentile of the means.
FY_D void k_noise_begin(const float* __restrict__ mean, NoiseCtl* __restrict__ ctl, long long n, double flat_pct,
                        double ref_intensity, unsigned long long A, unsigned long long B, unsigned long long step) {
    fy_pdl_wait();
    extern __shared__ unsigned int wsh[];                // 5 * 2048 counters
    const int t = threadIdx.x;
    const int c = (int)(n < kSampleMax ? n : kSampleMax);
    uint32_t k[kKeysPerThread];
    unsigned long long pos = (A * (unsigned long long)t + B) % (unsigned long long)n;   // step = A*kBoundThreads mod n
#pragma unroll
    for (int i = 0; i < kKeysPerThread; ++i) {
        k[i] = t + i * kBoundThreads < c ? fkey(__ldg(mean + pos)) : 0u;
        pos += step;
        if (pos >= (unsigned long long)n) pos -= (unsigned long long)n;
    }
    static_assert(sizeof(ctl->hist) % 16 == 0 && offsetof(NoiseCtl, hist) % 16 == 0, "uint4 clears");
    for (int i = t; i < (int)(sizeof(ctl->hist) / 16); i += kBoundThreads)
        reinterpret_cast<uint4*>(ctl->hist)[i] = make_uint4(0u, 0u, 0u, 0u);
    const double i1 = 1.0 / 100.0 * (double)(n - 1), i99 = 99.0 / 100.0 * (double)(n - 1);
    const long long k1 = (long long)i1, k99 = (long long)i99;
    if (t < NB) {
        target_init(ctl, t, t == 0 ? k1 : (t == 1 ? k99 : 0), n, t < 2);
        ctl->wbelow[t] = ctl->wvox[t] = ctl->bcount[t] = 0;
        ctl->ccnt[t] = ctl->bsn[t] = 0;
        ctl->wlo[t] = ctl->klo[t] = 0u;
        ctl->whi[t] = ctl->khi[t] = 0xffffffffu;
    }
    if (t == 0) {
        ctl->n = n;
        ctl->flat_pct = flat_pct;
        ctl->ref_intensity = ref_intensity;
        ctl->ntarget = 2;
        ctl->done_ctas = 0;
        ctl->ncand = 0;
        ctl->mode = kMeanWin;
    }
    if (c < 64) return;                                  // every key is a candidate
    const double nm = (double)(n > 1 ? n - 1 : 1);
    int lo0, hi0, lo1, hi1;
    window_ranks((double)k1 / nm, c, lo0, hi0);
    window_ranks((double)k99 / nm, c, lo1, hi1);
    const int rank[4] = {max(lo0, 0), min(hi0, c - 1), max(lo1, 0), min(hi1, c - 1)};
    uint32_t lo[4], hi[4];
    block_stats<4, false>(k, c, rank, wsh, lo, hi);
    if (t == 0) {
        ctl->klo[0] = lo[0]; ctl->khi[0] = hi[1];
        ctl->klo[1] = lo[2]; ctl->khi[1] = hi[3];
        if (lo0 >= 0) ctl->wlo[0] = lo[0];
        if (hi0 < c) ctl->whi[0] = hi[1];
        if (lo1 >= 0) ctl->wlo[1] = lo[2];
        if (hi1 < c) ctl->whi[1] = hi[3];
    }
}

// Buckets per target. The bins' windows hold nearly equal numbers of candidates (a bin's sample grows
// with it): at 512^3 60,000 to 700,000 each, so 300 to 6,000 keys a bucket.
constexpr int kMeanBuckets = 2048, kBinBuckets = 256;
static_assert(2 * kMeanBuckets <= kHist && NB * kBinBuckets <= kHist, "the control block's histogram holds them");

// The counting pass: mean keys against the windows of targets 0 and 1. The counts below each
// window stay in registers until one warp reduction at the end; the keys inside a window go
// to the candidate list (order is irrelevant to the selection). Per step a thread marks its
// 4*SU keys' window hits in two bit masks; one warp scan of the hit counts places them in the
// warp's shared-memory buffer, which is appended to the list (one atomic) when nearly full.
constexpr int kCountBuf = 1152;          // >= one step's worst case (32 lanes x 4*SU keys x 2); 45 KB static smem
FY_D void k_win_count(const float* __restrict__ mean, NoiseCtl* __restrict__ ctl,
                                                   float* __restrict__ cval, uint8_t* __restrict__ clab,
                                                   long long cap) {
    fy_pdl_wait();
    static_assert(32 * 4 * SU * 2 <= kCountBuf, "one step must fit the warp buffer");
    __shared__ float bufv[256 / 32][kCountBuf];
    __shared__ uint8_t bufl[256 / 32][kCountBuf];
    const unsigned full = 0xffffffffu;
    const int t = threadIdx.x, lane = t & 31;
    WarpCands wc;
    wc.v = bufv[t >> 5];
    wc.l = bufl[t >> 5];
    const long long n = ctl->n, n4 = (n + 3) / 4, n4f = n / 4;
    const uint32_t lo0 = ctl->wlo[0], hi0 = ctl->whi[0], lo1 = ctl->wlo[1], hi1 = ctl->whi[1];
    unsigned int bel0 = 0, bel1 = 0;
    const long long chunk = (long long)SU * 256;
    long long base = (long long)vbx() * chunk;
    const long long stride = (long long)vgx() * chunk;        // read once: the loop body has syncs
    // the next chunk's keys are loaded before this chunk's are used, so a warp keeps its loads
    // in flight while it classifies
    float4 xn[SU];
    if (base + chunk <= n4f) {
#pragma unroll
        for (int u = 0; u < SU; ++u) xn[u] = __ldg(reinterpret_cast<const float4*>(mean) + base + t + (long long)u * 256);
    }
    for (; base + chunk <= n4f; base += stride) {
        float4 x[SU];
#pragma unroll
        for (int u = 0; u < SU; ++u) x[u] = xn[u];
        if (base + stride + chunk <= n4f) {
#pragma unroll
            for (int u = 0; u < SU; ++u)
                xn[u] = __ldg(reinterpret_cast<const float4*>(mean) + base + stride + t + (long long)u * 256);
        }
        float mv[4 * SU];
        unsigned m0 = 0, m1 = 0;
#pragma unroll
        for (int u = 0; u < SU; ++u) {
            mv[4 * u] = x[u].x; mv[4 * u + 1] = x[u].y; mv[4 * u + 2] = x[u].z; mv[4 * u + 3] = x[u].w;
        }
#pragma unroll
        for (int q = 0; q < 4 * SU; ++q) {
            const uint32_t k = fkey(mv[q]);
            bel0 += k < lo0;
            bel1 += k < lo1;
            m0 |= (unsigned)(k >= lo0 && k <= hi0) << q;
            m1 |= (unsigned)(k >= lo1 && k <= hi1) << q;
        }
        const int c = __popc(m0) + __popc(m1);
        int incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(full, incl, o);
            if (lane >= o) incl += y;
        }
        const int tot = __shfl_sync(full, incl, 31);
        if (tot == 0) continue;
        if (wc.cnt + tot > kCountBuf) wc.flush(cval, clab, &ctl->ncand, cap);     // warp-uniform
        int pos = wc.cnt + incl - c;
#pragma unroll
        for (int q = 0; q < 4 * SU; ++q)          // unrolled, so mv stays in registers
            if ((m0 >> q) & 1u) { wc.v[pos] = mv[q]; wc.l[pos] = 0; ++pos; }
#pragma unroll
        for (int q = 0; q < 4 * SU; ++q)
            if ((m1 >> q) & 1u) { wc.v[pos] = mv[q]; wc.l[pos] = 1; ++pos; }
        wc.cnt += tot;
        __syncwarp();
    }
    if (base < n4) {                                     // the grid's partial chunk
        for (int u = 0; u < SU; ++u)
            for (int j = 0; j < 4; ++j) {
                const long long i = 4 * (base + t + (long long)u * 256) + j;
                if (i >= n) continue;
                const float mv = __ldg(mean + i);
                const uint32_t k = fkey(mv);
                bel0 += k < lo0;
                bel1 += k < lo1;
                for (int g = 0; g < 2; ++g)
                    if (k >= (g ? lo1 : lo0) && k <= (g ? hi1 : hi0)) {
                        const unsigned long long pos = atomicAdd(&ctl->ncand, 1ull);
                        if ((long long)pos < cap) { cval[pos] = mv; clab[pos] = (uint8_t)g; }
                    }
            }
    }
    wc.flush(cval, clab, &ctl->ncand, cap);
    const unsigned int s0 = __reduce_add_sync(full, bel0), s1 = __reduce_add_sync(full, bel1);
    if ((t & 31) == 0) {
        if (s0) atomicAdd(&ctl->wbelow[0], (unsigned long long)s0);
        if (s1) atomicAdd(&ctl->wbelow[1], (unsigned long long)s1);
    }
    if (!last_cta(ctl)) return;
    if (t < 2) window_buckets(ctl, t, kMeanBuckets);
    if (t == 0) {
        ctl->done_ctas = 0;
        if ((long long)__ldcg(&ctl->ncand) > cap || (noise_force_radix & 1)) ctl->mode = kMeanField;
    }
}

// f(value, target) for a thread's share of the candidates, U quads in flight at a time (collecting
// the bins' 39 MB of candidates at 512^3 takes 30 us with U = 1, 24 with 4; bucketing, whose shared
// atomics bound it, 24 with 1, 28 with 4).
template <int U, class F>
FY_D void for_each_cand(const NoiseCtl* __restrict__ ctl, const float* __restrict__ cval, const uint8_t* __restrict__ clab, F f) {
    const long long n = (long long)ctl->ncand, n4f = n / 4;
    const long long stride = (long long)vgx() * blockDim.x, i0 = (long long)vbx() * blockDim.x + threadIdx.x;
    for (long long q = i0; q < n4f; q += U * stride) {
        float4 x[U];
        uchar4 g[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (q + u * stride < n4f) {
                x[u] = *(reinterpret_cast<const float4*>(cval) + q + u * stride);
                g[u] = *(reinterpret_cast<const uchar4*>(clab) + q + u * stride);
            }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (q + u * stride < n4f) {
                f(x[u].x, g[u].x);
                f(x[u].y, g[u].y);
                f(x[u].z, g[u].z);
                f(x[u].w, g[u].w);
            }
    }
    for (long long i = 4 * n4f + i0; i < n; i += stride) f(cval[i], clab[i]);
}

// Bucket step for nt targets of nb buckets: the candidates' histogram; the last CTA finds per target the buckets
// of r = k - below and r + 1. `field` and `cand`: the modes of the radix passes that take over;
// force_bit: the test hook's bit for the latter; lcap: keys that a target can collect.
FY_D void cand_bucket(NoiseCtl* __restrict__ ctl, const float* __restrict__ cval, const uint8_t* __restrict__ clab, int nt,
                      int nb, long long lcap, int field, int cand, int force_bit) {
    extern __shared__ unsigned int rh[];
    __shared__ float sv0[NB], svs[NB];
    __shared__ int s_field, s_cand;
    const int t = threadIdx.x, lane = t & 31;
    const unsigned full = 0xffffffffu;
    for (int i = t; i < nt * nb; i += blockDim.x) rh[i] = 0;
    if (t < nt) { sv0[t] = ctl->cv0[t]; svs[t] = ctl->cvs[t]; }
    if (t == 0) s_field = s_cand = 0;
    __syncthreads();
    auto count = [&](float v, int g) { atomicAdd(&rh[g * nb + bucket_of(v, sv0[g], svs[g], nb)], 1u); };
    for_each_cand<1>(ctl, cval, clab, count);
    __syncthreads();
#pragma unroll 4
    for (int i = t; i < nt * nb; i += blockDim.x)
        if (rh[i]) atomicAdd(&ctl->hist[i], rh[i]);
    if (!last_cta(ctl)) return;
    const int forced = noise_force_radix & force_bit;
#pragma unroll 4
    for (int i = t; i < nt * nb; i += blockDim.x) {
        rh[i] = __ldcg(&ctl->hist[i]);
        ctl->hist[i] = 0;
    }
    __syncthreads();
    for (int g = t >> 5; g < nt; g += blockDim.x >> 5) {
        if (!ctl->tactive[g]) continue;
        const unsigned int* h = rh + g * nb;
        unsigned int total = 0;
        for (int i = lane; i < nb; i += 32) total += h[i];
        total = __reduce_add_sync(full, total);
        const long long k = ctl->tk[g], r = k - (long long)__ldcg(&ctl->wbelow[g]);
        const bool has_next = k + 1 < ctl->tgroup_n[g];
        if (!(r >= 0 && r < (long long)total && (!has_next || r + 1 < (long long)total))) {
            if (lane == 0) s_field = 1;
            continue;
        }
        int b0, b1;
        unsigned int before, before1;
        warp_find(h, nb, (unsigned)r, b0, before);
        b1 = b0;
        if (has_next) warp_find(h, nb, (unsigned)r + 1u, b1, before1);
        if (lane == 0) {
            const long long cnt = (long long)h[b0] + (b1 != b0 ? h[b1] : 0u);
            ctl->cb0[g] = b0;
            ctl->cb1[g] = b1;
            ctl->crank[g] = r - (long long)before;
            ctl->trank[g] = r;                            // for the radix passes over the candidates
            if (cnt > lcap || forced) s_cand = 1;
        }
    }
    __syncthreads();
    if (t < nt && s_field) ctl->trank[t] = ctl->tk[t];
    if (t == 0) {
        ctl->done_ctas = 0;
        if (s_field) ctl->mode = field;
        else if (s_cand) ctl->mode = cand;
    }
}

// Collect step: the candidates in their target's buckets into its list (the bucket step bounded
// their number by lcap). A CTA's hits wait in shared memory, so that each target's counter takes one
// atomic per CTA (one per key, 60,000 keys on 24 counters at 512^3, took 8 us more).
constexpr int kCollectBuf = 1024;
FY_D void cand_collect(NoiseCtl* __restrict__ ctl, const float* __restrict__ cval, const uint8_t* __restrict__ clab, int nt,
                       int nb, uint32_t* __restrict__ list, long long lcap) {
    __shared__ float sv0[NB], svs[NB];
    __shared__ int sb0[NB], sb1[NB];
    __shared__ unsigned int scnt[NB], sbase[NB], s_fill;
    __shared__ uint2 buf[kCollectBuf];                   // key; target << 16 | its place among the CTA's
    const int t = threadIdx.x;
    if (t < nt) {
        sv0[t] = ctl->cv0[t];
        svs[t] = ctl->cvs[t];
        sb0[t] = ctl->tactive[t] ? ctl->cb0[t] : -1;
        sb1[t] = ctl->tactive[t] ? ctl->cb1[t] : -1;
        scnt[t] = 0;
    }
    if (t == 0) s_fill = 0;
    __syncthreads();
    auto visit = [&](float v, int g) {
        const int b = bucket_of(v, sv0[g], svs[g], nb);
        if (b != sb0[g] && b != sb1[g]) return;
        const unsigned int f = atomicAdd(&s_fill, 1u);
        if (f < (unsigned)kCollectBuf) {
            buf[f] = make_uint2(fkey(v), (unsigned)g << 16 | atomicAdd(&scnt[g], 1u));
        } else {                                         // the buffer is full: straight to the list
            const unsigned int pos = atomicAdd(&ctl->ccnt[g], 1u);
            if (pos < lcap) list[g * lcap + pos] = fkey(v);
        }
    };
    for_each_cand<4>(ctl, cval, clab, visit);
    __syncthreads();
    if (t < nt && scnt[t]) sbase[t] = atomicAdd(&ctl->ccnt[t], scnt[t]);
    __syncthreads();
    const int fill = (int)min(s_fill, (unsigned)kCollectBuf);
    for (int i = t; i < fill; i += blockDim.x) {
        const unsigned int g = buf[i].y >> 16, pos = sbase[g] + (buf[i].y & 0xffffu);
        if (pos < lcap) list[g * lcap + pos] = buf[i].x;
    }
}
// Select step: one CTA per target selects the keys of k and k+1 among those collected.
FY_D void k_cand_select(NoiseCtl* __restrict__ ctl, const uint32_t* __restrict__ list, long long lcap, int win, int cand,
                        int used_bit) {
    fy_pdl_wait();
    extern __shared__ unsigned int wsh[];                // 3 * 2048 counters
    const int g = vbx(), t = threadIdx.x, mode = ctl->mode;
    if (t == 0 && g == 0 && (mode == win || mode == cand)) atomicOr(&noise_window_used, mode == cand ? used_bit * 5 : used_bit);
    if (mode != win || g >= ctl->ntarget || !ctl->tactive[g]) return;
    const int c = (int)ctl->ccnt[g], r = (int)ctl->crank[g];
    const bool has_next = ctl->tk[g] + 1 < ctl->tgroup_n[g];
    uint32_t k[kKeysPerThread];
#pragma unroll
    for (int i = 0; i < kKeysPerThread; ++i)
        k[i] = t + i * kBoundThreads < c ? list[g * lcap + t + i * kBoundThreads] : 0u;
    const int rank[2] = {r, has_next ? r + 1 : r};
    uint32_t lo[2], hi[2];
    block_stats<2, true>(k, c, rank, wsh, lo, hi);
    if (t == 0) {
        ctl->tprefix[g] = lo[0];
        ctl->tnext[g] = lo[1];
        ctl->tneed_next[g] = has_next;
        ctl->ccnt[g] = 0;
    }
}

FY_D void k_mean_bucket(NoiseCtl* __restrict__ ctl, const float* __restrict__ cval, const uint8_t* __restrict__ clab,
                        long long lcap) {
    fy_pdl_wait();
    if (ctl->mode == kMeanWin) cand_bucket(ctl, cval, clab, 2, kMeanBuckets, lcap, kMeanField, kMeanCand, 4);
}
FY_D void k_mean_collect(NoiseCtl* __restrict__ ctl, const float* __restrict__ cval, const uint8_t* __restrict__ clab,
                         uint32_t* __restrict__ list, long long lcap) {
    fy_pdl_wait();
    if (ctl->mode == kMeanWin) cand_collect(ctl, cval, clab, 2, kMeanBuckets, list, lcap);
}
FY_D void k_bin_bucket(NoiseCtl* __restrict__ ctl, const float* __restrict__ cval, const uint8_t* __restrict__ clab,
                       long long lcap) {
    fy_pdl_wait();
    if (ctl->mode == kBinWin) cand_bucket(ctl, cval, clab, NB, kBinBuckets, lcap, kBinField, kBinCand, 8);
}
FY_D void k_bin_collect(NoiseCtl* __restrict__ ctl, const float* __restrict__ cval, const uint8_t* __restrict__ clab,
                        uint32_t* __restrict__ list, long long lcap) {
    fy_pdl_wait();
    if (ctl->mode == kBinWin) cand_collect(ctl, cval, clab, NB, kBinBuckets, list, lcap);
}

// The bins: lo/hi from the selected means and the bin edges (noise.c:106-119), which every CTA
// forms for itself and one writes down; then the sample, each (mean, variance) pair's variance key
// listed under the bin of its mean (a CTA's keys of a bin take one atomic).
constexpr int kBinSampleThreads = 512;
FY_D void k_bin_sample(const float* __restrict__ mean, const float* __restrict__ var, NoiseCtl* __restrict__ ctl,
                       uint32_t* __restrict__ list, int lcap, long long m, unsigned long long A, unsigned long long B) {
    fy_pdl_wait();
    __shared__ float fe[NB + 1];
    __shared__ double s_lo, s_hi;
    __shared__ unsigned int scnt[NB], sbase[NB];
    const int t = threadIdx.x;
    const unsigned long long n = (unsigned long long)ctl->n;
    if (t == 0) {
        const double i1 = 1.0 / 100.0 * (double)(n - 1), i99 = 99.0 / 100.0 * (double)(n - 1);
        const long long k1 = (long long)i1, k99 = (long long)i99;
        const double lo = interp(ctl, 0, i1 - (double)k1, k1 + 1 < (long long)n);
        double hi = interp(ctl, 1, i99 - (double)k99, k99 + 1 < (long long)n);
        if (hi <= lo) hi = lo + 1e-6;                    // noise.c:109
        s_lo = lo;
        s_hi = hi;
    }
    if (t < NB) scnt[t] = 0;
    __syncthreads();
    if (t <= NB) {
        const double e = s_lo + (s_hi - s_lo) * t / NB;  // noise.c:118-119
        float f = (float)e;
        if ((double)f < e) f = nextafterf(f, INFINITY);
        fe[t] = f;
        if (vbx() == 0) {
            ctl->edge[t] = e;
            ctl->fedge[t] = f;
        }
    }
    if (vbx() == 0) {                                    // no CTA of this step reads these
        if (t < NB) ctl->wbelow[t] = ctl->wvox[t] = 0;
        if (t == 0) ctl->ncand = 0;
    }
    __syncthreads();
    const float lo_f = fe[0], fscale = (float)(NB / (s_hi - s_lo));
    const long long i = (long long)vbx() * blockDim.x + t;    // one sample per thread
    int b = -1;
    uint32_t key = 0;
    unsigned int pos = 0;
    if (i < m) {
        const unsigned long long q = (A * (unsigned long long)i + B) % n;
        const float mv = __ldg(mean + q), vv = __ldg(var + q);
        b = bin_of(mv, fe, lo_f, fscale);
        key = fkey(vv);
        if (b >= 0) pos = atomicAdd(&scnt[b], 1u);
    }
    __syncthreads();
    if (t < NB && scnt[t]) sbase[t] = atomicAdd(&ctl->bsn[t], scnt[t]);
    __syncthreads();
    if (b >= 0 && sbase[b] + pos < (unsigned)lcap) list[(size_t)b * lcap + sbase[b] + pos] = key;
}

// One CTA per bin: the window of its flat_pct percentile from its listed sample.
FY_D void k_bin_bounds(const uint32_t* __restrict__ list, int lcap, NoiseCtl* __restrict__ ctl) {
    fy_pdl_wait();
    extern __shared__ unsigned int wsh[];                // 3 * 2048 counters
    const int b = vbx(), t = threadIdx.x;
    const int c = (int)min(ctl->bsn[b], (unsigned)lcap);
    uint32_t k[kKeysPerThread];
#pragma unroll
    for (int i = 0; i < kKeysPerThread; ++i) k[i] = t + i * kBoundThreads < c ? list[(size_t)b * lcap + t + i * kBoundThreads] : 0u;
    uint32_t kl[2] = {0u, 0u}, kh[2] = {0xffffffffu, 0xffffffffu};
    int lo = -1, hi = c;
    if (c > 0) {
        if (c >= 64) window_ranks(ctl->flat_pct / 100.0, c, lo, hi);
        const int rank[2] = {min(max(lo, 0), c - 1), min(max(hi, 0), c - 1)};
        block_stats<2, false>(k, c, rank, wsh, kl, kh);
    }
    if (t == 0) {
        ctl->klo[b] = kl[0];
        ctl->khi[b] = kh[1];
        ctl->wlo[b] = lo >= 0 && lo < c ? kl[0] : 0u;             // no sample below (above): open
        ctl->whi[b] = hi >= 0 && hi < c ? kh[1] : 0xffffffffu;
    }
}

// The counting pass of the bins' windows: mean and variance read once, SUB float4 of each
// per thread and step. Every voxel takes the same branch-free path: its bin from the float
// guess (one 16-byte lookup gives the guessed bin's edges and window; when the mean lies outside
// the guess, by rounding at an edge or in a degenerate range, the exact walk corrects it), the
// key of its variance against the bin's window, and one read-modify-write of the lane's own
// shared-memory counter of its bin (low 16 bits: the bin's voxels, high 16 bits: those below the
// window; rows of 25 words, so the lanes of a warp hit distinct banks when they share a bin;
// added into the CTA's totals before a field can pass 65535). The keys inside the window are
// placed by one warp scan per step in the warp's buffer and appended to the list (one atomic per
// buffer), as in k_win_count. The last CTA sets the bins' ranks from the counts.
constexpr int kBCountBuf = 512;          // per warp: two steps' worst case (32 x 8 each)
constexpr int kLaneRow = 25;             // counter words per lane (NB = 24, odd stride)
FY_D void k_bwin_count(const float* __restrict__ mean, const float* __restrict__ var,
                                                       NoiseCtl* __restrict__ ctl, float* __restrict__ cval,
                                                       uint8_t* __restrict__ clab, long long cap) {
    fy_pdl_wait();
    constexpr int SUB = 2;                               // float4 of each field per thread and step
    static_assert(32 * 4 * SUB <= kBCountBuf && NB < kLaneRow, "buffer and counter rows");
    __shared__ float bufv[256 / 32][kBCountBuf];
    __shared__ uint8_t bufl[256 / 32][kBCountBuf];
    __shared__ unsigned int lc[256 * kLaneRow];          // per-lane counters
    __shared__ float fe[NB + 1];
    __shared__ float4 stab[NB];                          // per bin: its edges and its window
    __shared__ unsigned int sc[NB * 2];
    const unsigned full = 0xffffffffu;
    const int t = threadIdx.x, lane = t & 31;
    if (t <= NB) fe[t] = ctl->fedge[t];
    if (t < NB)
        stab[t] = make_float4(ctl->fedge[t], ctl->fedge[t + 1], __uint_as_float(ctl->wlo[t]), __uint_as_float(ctl->whi[t]));
    for (int i = t; i < NB * 2; i += blockDim.x) sc[i] = 0;
    for (int i = t; i < 256 * kLaneRow; i += blockDim.x) lc[i] = 0;
    __syncthreads();
    const float lo_e = fe[0], hi_e = fe[NB], fscale = (float)(NB / (ctl->edge[NB] - ctl->edge[0]));
    unsigned int* row = lc + t * kLaneRow;
    WarpCands wc;
    wc.v = bufv[t >> 5];
    wc.l = bufl[t >> 5];
    // bin (or -1 outside every bin) and whether the key is inside the bin's window
    auto classify = [&](float m, float v, bool valid, int& bo, bool& inside) {
        const bool inr = valid && m >= lo_e && m < hi_e;
        const float mc = inr ? m : lo_e;
        int b = (int)((mc - lo_e) * fscale);
        b = b < 0 ? 0 : (b > NB - 1 ? NB - 1 : b);
        float4 e = stab[b];
        if (!(mc >= e.x && mc < e.y)) {
            b = max(bin_of(mc, fe, lo_e, fscale), 0);
            e = stab[b];
        }
        const uint32_t k = fkey(v), wl = __float_as_uint(e.z), wh = __float_as_uint(e.w);
        row[b] += inr ? (k < wl ? 0x10001u : 1u) : 0u;
        inside = inr && k >= wl && k <= wh;
        bo = b;
    };
    auto flush_rows = [&]() {                             // CTA-uniform
        __syncthreads();
        if (lane < NB) {                                 // lane = bin, each warp its own 32 rows
            unsigned int vox = 0, below = 0;
#pragma unroll 8
            for (int l = t & ~31; l < (t & ~31) + 32; ++l) {
                const unsigned int w = lc[l * kLaneRow + lane];
                vox += w & 0xffffu;
                below += w >> 16;
            }
            if (vox) atomicAdd(&sc[2 * lane], vox);
            if (below) atomicAdd(&sc[2 * lane + 1], below);
        }
        __syncthreads();
        for (int i = 0; i < NB; ++i) row[i] = 0;
        __syncthreads();
    };
    const long long n = ctl->n, n4 = (n + 3) / 4, n4f = n / 4;
    const long long chunk = (long long)SUB * 256;
    long long base = (long long)vbx() * chunk;
    const long long stride = (long long)vgx() * chunk;        // read once: the loop body has syncs
    int steps = 0;
    for (; base + chunk <= n4f; base += stride) {
        float4 xm[SUB], xv[SUB];
#pragma unroll
        for (int u = 0; u < SUB; ++u) {
            const long long q = base + (long long)t * SUB + u;
            xm[u] = __ldg(reinterpret_cast<const float4*>(mean) + q);
            xv[u] = __ldg(reinterpret_cast<const float4*>(var) + q);
        }
        float vv[4 * SUB];
        int bq[4 * SUB];
        unsigned hit = 0;
#pragma unroll
        for (int u = 0; u < SUB; ++u) {
            const float mm[4] = {xm[u].x, xm[u].y, xm[u].z, xm[u].w};
            vv[4 * u] = xv[u].x; vv[4 * u + 1] = xv[u].y; vv[4 * u + 2] = xv[u].z; vv[4 * u + 3] = xv[u].w;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                bool ins;
                classify(mm[j], vv[4 * u + j], true, bq[4 * u + j], ins);
                hit |= (unsigned)ins << (4 * u + j);
            }
        }
        if (++steps == 65535 / (4 * SUB)) {              // a 16-bit field could pass 65535
            flush_rows();
            steps = 0;
        }
        const int c = __popc(hit);
        int incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(full, incl, o);
            if (lane >= o) incl += y;
        }
        const int tot = __shfl_sync(full, incl, 31);
        if (tot == 0) continue;
        if (wc.cnt + tot > kBCountBuf) wc.flush(cval, clab, &ctl->ncand, cap);     // warp-uniform
        int pos = wc.cnt + incl - c;
#pragma unroll
        for (int q = 0; q < 4 * SUB; ++q)
            if ((hit >> q) & 1u) { wc.v[pos] = vv[q]; wc.l[pos] = (uint8_t)bq[q]; ++pos; }
        wc.cnt += tot;
        __syncwarp();
    }
    if (base < n4) {                                      // the grid's partial chunk (CTA-uniform)
        for (int u = 0; u < SUB; ++u)
            for (int j = 0; j < 4; ++j) {
                const long long i = 4 * (base + (long long)t * SUB + u) + j;
                const bool valid = i < n;
                const float v = valid ? __ldg(var + i) : 0.f;
                int b;
                bool ins;
                classify(valid ? __ldg(mean + i) : 0.f, v, valid, b, ins);
                if (ins) {
                    const unsigned long long pos = atomicAdd(&ctl->ncand, 1ull);
                    if ((long long)pos < cap) { cval[pos] = v; clab[pos] = (uint8_t)b; }
                }
            }
    }
    wc.flush(cval, clab, &ctl->ncand, cap);
    flush_rows();
    if (t < NB) {
        if (sc[2 * t]) atomicAdd(&ctl->wvox[t], (unsigned long long)sc[2 * t]);
        if (sc[2 * t + 1]) atomicAdd(&ctl->wbelow[t], (unsigned long long)sc[2 * t + 1]);
    }
    if (!last_cta(ctl)) return;
    // the targets: the flat_pct percentile of every bin of >= 200 voxels (noise.c:123), or of all
    // variances when no bin has them (noise.c:166-171)
    if (t >= 32) return;
    long long cnt = 0;
    if (t < NB) {
        cnt = (long long)__ldcg(&ctl->wvox[t]);
        ctl->bcount[t] = (unsigned long long)cnt;
    }
    const bool on = cnt >= 200, any = __any_sync(full, on);
    if (t < NB) {
        if (any) target_init(ctl, t, on ? (long long)(ctl->flat_pct / 100.0 * (double)(cnt - 1)) : 0, cnt, on);
        else target_init(ctl, t, t == 0 ? (long long)(ctl->flat_pct / 100.0 * (double)(n - 1)) : 0, n, t == 0);
    }
    if (t < NB) window_buckets(ctl, t, kBinBuckets);
    if (t == 0) {
        ctl->done_ctas = 0;
        ctl->ntarget = any ? NB : 1;
        ctl->mode = !any ? kVarField
                         : ((long long)__ldcg(&ctl->ncand) > cap || (noise_force_radix & 2) ? kBinField : kBinWin);
    }
}

// IRLS fit (FP64) and outputs. One warp: lane b handles bin b, so the bins' loads are in flight
// together. The used bins are compacted in bin order; the weights, residuals and the median of the
// residuals are formed by one lane per bin, the five weighted sums by lane 0 in the reference's
// order (noise.c:141-147), so every value equals the sequential fit's.
FY_D void k_noise_fit(NoiseCtl* ctl) {
    fy_pdl_wait();
    static_assert(NB <= 32, "one lane per bin");
    const int lane = threadIdx.x;
    __shared__ double s_i[NB], s_f[NB], s_w[NB], s_r[NB], s_one[NB];
    __shared__ long long s_c[NB];
    __shared__ double s_g, s_b;
    __shared__ int s_brk;
    const unsigned full = 0xffffffffu;
    const bool in_use = lane < NB && (long long)ctl->bcount[lane] >= 200;
    if (lane < NB) s_one[lane] = 1.0;
    const unsigned um = __ballot_sync(full, in_use);
    const int used = __popc(um);
    if (in_use) {
        const int pos = __popc(um & ((1u << lane) - 1u));
        s_c[pos] = (long long)ctl->bcount[lane];
        s_i[pos] = 0.5 * (ctl->edge[lane] + ctl->edge[lane + 1]);
        const double idx = ctl->flat_pct / 100.0 * (double)(s_c[pos] - 1);
        const long long k = (long long)idx;
        s_f[pos] = interp(ctl, lane, idx - (double)k, k + 1 < s_c[pos]);     // the bin's floor
    }
    __syncwarp();
    double g = 0, bb = 0;
    if (lane == 0) ctl->out_used = used;
    if (ctl->mode == kVarField) {
        if (lane == 0) {
            const long long n = ctl->n;
            const double idx = ctl->flat_pct / 100.0 * (double)(n - 1);
            const long long k = (long long)idx;
            bb = interp(ctl, 0, idx - (double)k, k + 1 < n);
        }
    } else if (used >= 3) {                               // IRLS, noise.c:139-161
        if (lane < used) s_w[lane] = sqrt((double)s_c[lane]);
        __syncwarp();
        for (int it = 0; it < 4; it++) {
            // the five weighted sums, one lane each, in the reference's order (noise.c:141-147):
            // Sw += w, Swx += w*x, Swy += w*y, Swxx += w*x*x, Swxy += w*x*y (the factors that a sum
            // lacks are 1; one lane doing all five took 7 us in all, lanes in five branches 27)
            const double* f1 = lane == 0 ? s_one : (lane == 2 ? s_f : s_i);
            const double* f2 = lane == 3 ? s_i : (lane == 4 ? s_f : s_one);
            double acc = 0;
            for (int i = 0; i < used; i++) acc += s_w[i] * f1[i] * f2[i];
            const double Sw = __shfl_sync(full, acc, 0), Swx = __shfl_sync(full, acc, 1), Swy = __shfl_sync(full, acc, 2);
            const double Swxx = __shfl_sync(full, acc, 3), Swxy = __shfl_sync(full, acc, 4);
            if (lane == 0) {
                const double det = Sw * Swxx - Swx * Swx;
                s_brk = fabs(det) < 1e-20;
                if (!s_brk) {
                    s_g = (Sw * Swxy - Swx * Swy) / det;
                    s_b = (Swxx * Swy - Swx * Swxy) / det;
                }
            }
            __syncwarp();
            if (s_brk) break;
            g = s_g;
            bb = s_b;
            double res = 0.0;
            if (lane < used) {
                res = fabs(s_f[lane] - (g * s_i[lane] + bb));
                s_r[lane] = res;
            }
            __syncwarp();
            // percentile(resid, used, 50) (noise.c:66-73): the values at sorted positions lo and
            // lo + 1, found by ranking each residual (ties by index)
            const double pidx = 50.0 / 100.0 * (used - 1);
            const int plo = (int)pidx;
            const double pf = pidx - plo;
            int rank = 0;
            if (lane < used)
                for (int j = 0; j < used; ++j) rank += s_r[j] < res || (s_r[j] == res && j < lane);
            const unsigned mlo = __ballot_sync(full, lane < used && rank == plo);
            const unsigned mhi = __ballot_sync(full, lane < used && rank == plo + 1);
            const double vlo = __shfl_sync(full, res, mlo ? __ffs(mlo) - 1 : 0);    // (no rank: NaN residuals)
            const double vhi = __shfl_sync(full, res, mhi ? __ffs(mhi) - 1 : (mlo ? __ffs(mlo) - 1 : 0));
            const double med = (plo + 1 < used ? vlo * (1 - pf) + vhi * pf : vlo) + 1e-9;
            if (lane < used) {
                const double rr = res / (2.0 * med);
                s_w[lane] = sqrt((double)s_c[lane]) / (1.0 + rr * rr);
            }
            __syncwarp();
        }
    } else if (used > 0) {                                // noise.c:162-165
        if (lane == 0) {
            double sum = 0;
            for (int i = 0; i < used; i++) sum += s_f[i];
            bb = sum / used;
        }
    }
    if (lane != 0) return;
    if (!isfinite(g)) g = 0;
    if (!isfinite(bb)) bb = 0;
    double var_ref = g * ctl->ref_intensity + bb;
    if (var_ref < 0) var_ref = bb > 0 ? bb : 0;
    const double noise_ref = sqrt(var_ref) * 1.15;      // noise.c:181-187
    ctl->out_g = g; ctl->out_b = bb;
    ctl->out_noise_ref = noise_ref;
    ctl->out_ref_intensity = ctl->ref_intensity;
    double eps = (3.0 * noise_ref) * (3.0 * noise_ref);  // noise.c:197-202
    if (!(eps > 1e-8)) eps = 1e-8;
    ctl->eps = (float)eps;
}

unsigned grid_sel(long long n, int sms) {
    long long g = (n / 4 + 256 * SU - 1) / (256 * SU);
    const long long cap = (long long)sms * 8;
    return (unsigned)(g < cap ? (g ? g : 1) : cap);
}

}  // namespace

size_t fy_noise_ctl_bytes() { return (sizeof(NoiseCtl) + 255) & ~(size_t)255; }

namespace {
// Scratch layout (floats; every sub-array 256-byte aligned for the vector loads): mean, var, bin
// labels (bytes; before the radix passes over the bins they hold the collected keys), the bins'
// sample lists, and the candidate list (values, then labels) of capacity n/8 + 4096 (the windows
// hold a few percent of the voxels).
size_t round64(size_t v) { return (v + 63) & ~(size_t)63; }
struct NoiseLayout {
    size_t mean, var, bin, samp, cval, clab, total;
    long long cap;
};
NoiseLayout noise_layout(size_t n) {
    NoiseLayout L;
    const size_t nr = round64(n);
    L.mean = 0;
    L.var = nr;
    L.bin = 2 * nr;
    L.samp = L.bin + round64((n + 3) / 4);
    L.cap = (long long)((n + 7) / 8 + 4096);
    L.cval = L.samp + (size_t)NB * kBinListSmall;
    L.clab = L.cval + round64((size_t)L.cap);
    L.total = L.clab + round64(((size_t)L.cap + 3) / 4);
    return L;
}
// Weyl step for the sample positions: a prime a with gcd(a, n) = 1, reduced mod n (for a
// prime a that means n < a, or a not dividing n).
unsigned long long weyl_step(unsigned long long n) {
    if (n <= 1) return 1;
    const unsigned long long primes[4] = {2654435761ull, 2246822519ull, 3266489917ull, 668265263ull};
    for (unsigned long long a : primes)
        if (n < a || n % a != 0) return a % n;
    return 1;
}
}  // namespace

size_t fy_noise_scratch_floats(size_t n) { return noise_layout(n).total; }

// The statistics pass's parameters for one volume, rows of `in` in_pitch floats apart (0: nx): mean and
// variance fields dense in the scratch, the guided (mean, var) pairs (optional) in rows of fy_pitch(nx).
fyzb::Params fy_noise_stats_params(const float* in, int nz, int ny, int nx, int win, float* scratch, float* guided_mv,
                                   int in_pitch) {
    const NoiseLayout Lay = noise_layout((size_t)nz * ny * nx);
    fyzb::Params sp{};
    sp.nz = nz; sp.ny = ny; sp.nx = nx;
    sp.f0 = in; sp.o0 = scratch + Lay.mean; sp.o1 = scratch + Lay.var; sp.o2 = guided_mv;
    sp.inv_wc = (float)(1.0 / ((double)win * win * win));
    sp.wci = win * win * win;
    sp.pf0 = in_pitch;
    sp.pmv = fy_pitch(nx);
    return sp;
}

namespace {

// ---------------------------------------------------------------- launching: one cube or a batch
// Every selection step above is a __device__ body run by one of two wrappers: k_one, one volume,
// the body's arguments as kernel parameters; k_many, a batch of volumes, the CTA's volume from
// its block index
// and each volume's arguments read from a device array. NoiseLaunch either launches k_one at
// once or, in batch mode, records each volume's arguments and grid for every step of the
// sequence (the same sequence for every volume) and then replays it: one launch per step for
// all volumes, each volume with the CTAs it asked for (their blocks are numbered per volume
// through vbx()/vgx(); the grids that index targets or bins along y are the same for all).
template <int NTB, int MINB, auto F, class... P>
__global__ void __launch_bounds__(NTB, MINB) k_one(P... a) {
    s_vbx = blockIdx.x;                    // every thread stores the same values
    s_vgx = gridDim.x;
    F(a...);
}
// prefix[v] = the first CTA (along x) of volume v, prefix[nvol] = all of them
template <int NTB, int MINB, auto F, class... P>
__global__ void __launch_bounds__(NTB, MINB) k_many(const cuda::std::tuple<P...>* __restrict__ packs,
                                                     const unsigned* __restrict__ prefix, int nvol) {
    int lo = 0, hi = nvol - 1;             // the last volume whose first CTA <= blockIdx.x
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(prefix + mid) <= blockIdx.x) lo = mid; else hi = mid - 1;
    }
    s_vbx = blockIdx.x - __ldg(prefix + lo);
    s_vgx = __ldg(prefix + lo + 1) - __ldg(prefix + lo);
    cuda::std::apply([](auto... x) { F(x...); }, packs[lo]);
}

struct NoiseLaunch {
    cudaStream_t st = nullptr;
    bool record = false;
    struct Step {
        const void* kern;                  // the k_many instance
        dim3 grid, block;
        size_t smem, pack;                 // bytes of one volume's arguments
        std::vector<unsigned char> packs;
        std::vector<unsigned> gx;         // CTAs along x of each volume
    };
    std::vector<Step> steps;
    size_t si = 0;                         // the next step of the volume being recorded
    int cubes = 0;

    template <int NTB, int MINB, auto F, class... P, class... A>
    cudaError_t run_sig(void (*)(P...), dim3 grid, dim3 block, size_t smem, A... a) {
        if (!record) {
            auto k = k_one<NTB, MINB, F, P...>;
            cudaError_t e = fy_smem_optin(k, smem);
            if (e != cudaSuccess) return e;
            return fy_launch_pdl(k, grid, block, smem, st, (P)a...);
        }
        using T = cuda::std::tuple<P...>;
        const void* k = (const void*)k_many<NTB, MINB, F, P...>;
        if (si == steps.size()) {
            if (cubes > 0) return cudaErrorInvalidValue;          // every volume has the same sequence
            cudaError_t e = fy_smem_optin(k_many<NTB, MINB, F, P...>, smem);
            if (e != cudaSuccess) return e;
            steps.push_back(Step{k, grid, block, smem, sizeof(T), {}});
        }
        Step& s = steps[si++];
        if (s.kern != k || s.block.x != block.x || s.smem != smem) return cudaErrorInvalidValue;
        if (s.grid.y != grid.y) return cudaErrorInvalidValue;
        s.gx.push_back(grid.x);
        const T t((P)a...);
        const unsigned char* b = reinterpret_cast<const unsigned char*>(&t);
        s.packs.insert(s.packs.end(), b, b + sizeof(T));
        return cudaSuccess;
    }
    template <int NTB, int MINB, auto F, class... A>
    cudaError_t run(dim3 grid, dim3 block, size_t smem, A... a) {
        return run_sig<NTB, MINB, F>(F, grid, block, smem, a...);
    }
};

#define RUN(NTB, MINB, F, ...)                                                 \
    do {                                                                       \
        const cudaError_t pe_ = L.run<NTB, MINB, F>(__VA_ARGS__);              \
        if (pe_ != cudaSuccess) return pe_;                                    \
        ++launches;                                                            \
    } while (0)

// The estimate's launch sequence for one volume through L. stats: run the statistics pass here
// (a batch runs it for all volumes at once before the sequence).
cudaError_t noise_sequence(NoiseLaunch& L, const float* in, int nz, int ny, int nx, int win, double flat_pct,
                           double ref_intensity, float* scratch, void* ctl_mem, int sms, int& launches,
                           float* guided_mv, bool stats, int in_pitch = 0) {
    cudaStream_t st = L.st;
    NoiseCtl* ctl = (NoiseCtl*)ctl_mem;
    const long long n = (long long)nz * ny * nx;
    const NoiseLayout Lay = noise_layout((size_t)n);
    float* mean = scratch + Lay.mean;
    float* var = scratch + Lay.var;
    uint8_t* bin = (uint8_t*)(scratch + Lay.bin);
    uint32_t* keys = (uint32_t*)(scratch + Lay.bin);
    float* cval = scratch + Lay.cval;
    uint8_t* clab = (uint8_t*)(scratch + Lay.clab);
    const unsigned g = grid_sel(n, sms), gc = grid_sel(Lay.cap, sms);
    // Passes that usually exit at once (the radix passes): few and large CTAs, so the common case
    // schedules few empty ones; when they do run, their grid-stride loops cover every voxel. What bounds
    // them then is latency (means: two CTAs of 512 threads per SM 262 us a pass over 512^3, one of 256
    // 436) and the CTAs' histograms joining the field's (bins of one value each, 512^3, four passes:
    // one CTA of 1024 threads per SM 1410 us, four of 256 2000, four of 512 1999). In a batch, where every
    // volume brings its CTAs, small ones exit faster: 16 cubes of 96..128 take 947 us so and 994 us
    // with the large ones.
    auto per_sm = [&](unsigned k, unsigned threads) {     // k CTAs per SM, fewer where a step covers the field
        const unsigned steps = (g * 256 + threads - 1) / threads;
        return steps < k * (unsigned)sms ? steps : k * (unsigned)sms;
    };
    // candidate lists hold a few percent of the voxels (their capacity is n/8): two CTAs per SM
    const unsigned gcl = (unsigned)(gc < 2u * (unsigned)sms ? gc : 2u * (unsigned)sms);
    const size_t smem_hist = kHist * sizeof(unsigned int);
    const unsigned long long wa = weyl_step((unsigned long long)n);
    // keys that a target can collect: the label region holds n/4 words
    const long long lc_mean = n / 8 < kListMax ? n / 8 : kListMax, lc_bin = n / (4 * NB) < kListMax ? n / (4 * NB) : kListMax;
    const size_t smem_stats = 2048 * sizeof(unsigned int);
    if (stats) {   // 1. stats
        cudaError_t e0 = fyzb::launch<fyzb::ZB_NOISE>(fy_noise_stats_params(in, nz, ny, nx, win, scratch, guided_mv, in_pitch),
                                                      win / 2, sms, st);
        if (e0 != cudaSuccess) return e0;
        ++launches;
        if (!L.record) fy_prof_mark(st, "noise.stats");
    }
    // 2. the 1st/99th percentile of the means: window steps, then the radix passes behind them
    RUN(kBoundThreads, 1, k_noise_begin, 1, kBoundThreads, 5 * smem_stats, mean, ctl, n, flat_pct, ref_intensity, wa,
        (unsigned long long)n / 3, (wa * (unsigned long long)kBoundThreads) % (unsigned long long)n);
    RUN(256, 3, k_win_count, g, 256, 0, mean, ctl, cval, clab, Lay.cap);
    RUN(512, 1, k_mean_bucket, gcl, 512, smem_hist, ctl, cval, clab, lc_mean);
    RUN(256, 1, k_mean_collect, gcl, 256, 0, ctl, cval, clab, keys, lc_mean);
    RUN(kBoundThreads, 1, k_cand_select, 2, kBoundThreads, 3 * smem_stats, ctl, keys, lc_mean, (int)kMeanWin, (int)kMeanCand, 1);
    for (int sh = 24; sh >= 0; sh -= 8) {
        if (L.record) RUN(256, 1, k_mean_radix, per_sm(1, 256), 256, smem_hist, mean, ctl, cval, clab, sh);
        else RUN(512, 1, k_mean_radix, per_sm(2, 512), 512, smem_hist, mean, ctl, cval, clab, sh);
    }
    if (!L.record) fy_prof_mark(st, "noise.lohi");
    // the per-bin flat_pct percentile of the variance, the same way. The sample lists use the
    // candidate region when it is large enough (the counting pass refills it afterwards).
    {
        long long m2 = n < kBinSampleMax ? n : kBinSampleMax;
        const bool large = Lay.cap >= 2 * (long long)NB * kBinListSmall;
        uint32_t* slist = large ? (uint32_t*)cval : (uint32_t*)(scratch + Lay.samp);
        const int scap = !large ? kBinListSmall : (Lay.cap / NB < kBinListMax ? (int)(Lay.cap / NB) : kBinListMax);
        RUN(kBinSampleThreads, 1, k_bin_sample, (unsigned)((m2 + kBinSampleThreads - 1) / kBinSampleThreads), kBinSampleThreads, 0,
            mean, var, ctl, slist, scap, m2, wa, (unsigned long long)n / 5);
        RUN(kBoundThreads, 1, k_bin_bounds, NB, kBoundThreads, 3 * smem_stats, slist, scap, ctl);
        RUN(256, 4, k_bwin_count, g, 256, 0, mean, var, ctl, cval, clab, Lay.cap);
        RUN(512, 1, k_bin_bucket, gcl, 512, smem_hist, ctl, cval, clab, lc_bin);
        RUN(256, 1, k_bin_collect, gcl, 256, 0, ctl, cval, clab, keys, lc_bin);
        RUN(kBoundThreads, 1, k_cand_select, NB, kBoundThreads, 3 * smem_stats, ctl, keys, lc_bin, (int)kBinWin, (int)kBinCand, 2);
    }
    for (int sh = 24; sh >= 0; sh -= 8) {
        if (L.record) RUN(256, 1, k_bin_radix, per_sm(4, 256), 256, smem_hist, mean, var, bin, ctl, cval, clab, sh);
        else RUN(1024, 1, k_bin_radix, per_sm(1, 1024), 1024, smem_hist, mean, var, bin, ctl, cval, clab, sh);
    }
    RUN(32, 1, k_noise_fit, 1, 32, 0, ctl);
    if (!L.record) fy_prof_mark(st, "noise.bin_select");
    return cudaSuccess;
}

}  // namespace

// Enqueue the whole estimate. scratch: fy_noise_scratch_floats(n) floats; ctl:
// fy_noise_ctl_bytes(). Supports win in {3..9} (r = win/2 <= 4). guided_mv (optional,
// fy_guided_fused_scratch_floats, rows fy_pitch(nx) voxels apart): the statistics pass also writes the guided filter's (mean, var) pairs of the
// same window, for fy_launch_guided_apply_mv with r = win/2. in_pitch: floats per row of `in` (0: nx).
// Every kernel runs as a programmatic dependent launch; the first failed launch is returned.
cudaError_t fy_launch_estimate_noise(const float* in, int nz, int ny, int nx, int win, double flat_pct,
                                     double ref_intensity, float* scratch, void* ctl_mem, int sms,
                                     cudaStream_t st, int& launches, float* guided_mv, int in_pitch) {
    NoiseLaunch L;
    L.st = st;
    cudaError_t e = noise_sequence(L, in, nz, ny, nx, win, flat_pct, ref_intensity, scratch, ctl_mem, sms, launches,
                                   guided_mv, true, in_pitch);
    return e != cudaSuccess ? e : cudaGetLastError();
}

// ---------------------------------------------------------------- a batch of volumes
// The selection sequences of many volumes, recorded (no launch) for one replay: each step of
// the sequence becomes one launch over all volumes' CTAs. The statistics pass
// is not part of it (the caller runs it for every volume first: fy_noise_stats_params).
struct NoiseBatch {
    NoiseLaunch L;
    int launches = 0;                      // per volume
};
NoiseBatch* fy_noise_batch_record(const float* const* in, const int* dims, float* const* scratch,
                                  void* const* ctl_mem, int nvol, int win, double flat_pct, double ref_intensity,
                                  int sms, cudaError_t* err) {
    NoiseBatch* b = new NoiseBatch();
    b->L.record = true;
    *err = cudaSuccess;
    for (int i = 0; i < nvol && *err == cudaSuccess; ++i) {
        int launches = 0;
        b->L.si = 0;
        *err = noise_sequence(b->L, in[i], dims[3 * i], dims[3 * i + 1], dims[3 * i + 2], win, flat_pct, ref_intensity,
                              scratch[i], ctl_mem[i], sms, launches, nullptr, false);
        if (*err == cudaSuccess && b->L.si != b->L.steps.size()) *err = cudaErrorInvalidValue;
        b->L.cubes = i + 1;
        b->launches = launches;
    }
    if (*err != cudaSuccess) {
        delete b;
        return nullptr;
    }
    return b;
}
// Bytes of the packed steps: per step its volumes' arguments, then its table of first CTAs per
// volume (nvol + 1 entries), each 256-byte aligned.
static size_t al256n(size_t v) { return (v + 255) & ~(size_t)255; }
size_t fy_noise_batch_bytes(const NoiseBatch* b) {
    size_t t = 0;
    for (const auto& s : b->L.steps) t += al256n(s.packs.size()) + al256n((s.gx.size() + 1) * sizeof(unsigned));
    return t;
}
void fy_noise_batch_pack(const NoiseBatch* b, void* host) {
    unsigned char* h = (unsigned char*)host;
    for (const auto& s : b->L.steps) {
        memcpy(h, s.packs.data(), s.packs.size());
        h += al256n(s.packs.size());
        unsigned* pre = reinterpret_cast<unsigned*>(h);
        pre[0] = 0;
        for (size_t v = 0; v < s.gx.size(); ++v) pre[v + 1] = pre[v] + s.gx[v];
        h += al256n((s.gx.size() + 1) * sizeof(unsigned));
    }
}
int fy_noise_batch_steps(const NoiseBatch* b) { return (int)b->L.steps.size(); }
// One launch per step on st, its volumes' arguments read from dev (fy_noise_batch_pack's
// layout, already in device memory by stream order).
cudaError_t fy_noise_batch_launch(const NoiseBatch* b, const void* dev, cudaStream_t st) {
    const unsigned char* d = (const unsigned char*)dev;
    for (const auto& s : b->L.steps) {
        unsigned total = 0;
        for (unsigned g : s.gx) total += g;
        const void* packs = d;
        d += al256n(s.packs.size());
        const void* prefix = d;
        d += al256n((s.gx.size() + 1) * sizeof(unsigned));
        int nvol = b->L.cubes;
        cudaLaunchConfig_t c = {};
        c.gridDim = dim3(total, s.grid.y, 1);
        c.blockDim = s.block;
        c.dynamicSmemBytes = s.smem;
        c.stream = st;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
        c.attrs = at;
        c.numAttrs = 1;
        void* args[3] = {(void*)&packs, (void*)&prefix, (void*)&nvol};
        cudaError_t e = cudaLaunchKernelExC(&c, s.kern, args);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}
void fy_noise_batch_free(NoiseBatch* b) { delete b; }
// Copy the model out of a finished control block (device -> host, async on st).
cudaError_t fy_noise_read(const void* ctl_mem, double* g, double* b, double* noise_ref, double* ref_intensity,
                          int* used, cudaStream_t st) {
    static_assert(sizeof(double) == 8, "");
    const NoiseCtl* ctl = (const NoiseCtl*)ctl_mem;
    cudaError_t e;
    if ((e = cudaMemcpyAsync(g, &ctl->out_g, 8, cudaMemcpyDeviceToHost, st))) return e;
    if ((e = cudaMemcpyAsync(b, &ctl->out_b, 8, cudaMemcpyDeviceToHost, st))) return e;
    if ((e = cudaMemcpyAsync(noise_ref, &ctl->out_noise_ref, 8, cudaMemcpyDeviceToHost, st))) return e;
    if ((e = cudaMemcpyAsync(ref_intensity, &ctl->out_ref_intensity, 8, cudaMemcpyDeviceToHost, st))) return e;
    return cudaMemcpyAsync(used, &ctl->out_used, 4, cudaMemcpyDeviceToHost, st);
}

const float* fy_noise_eps_ptr(const void* ctl_mem) { return &((const NoiseCtl*)ctl_mem)->eps; }

namespace {
// One thread copies a finished model into caller device memory laid out as fy_noise_model.
__global__ void k_noise_store(const NoiseCtl* __restrict__ ctl, fy_noise_model* __restrict__ m,
                              float* __restrict__ eps) {
    m->g = ctl->out_g;
    m->b = ctl->out_b;
    m->noise_ref = ctl->out_noise_ref;
    m->ref_intensity = ctl->out_ref_intensity;
    m->n_bins_used = ctl->out_used;
    if (eps) *eps = ctl->eps;
}
}  // namespace

cudaError_t fy_noise_store(const void* ctl_mem, void* d_model, float* d_eps, cudaStream_t st) {
    k_noise_store<<<1, 1, 0, st>>>((const NoiseCtl*)ctl_mem, (fy_noise_model*)d_model, d_eps);
    return cudaGetLastError();
}

// Test hook of the selection paths (see noise_force_radix): sets the forcing mask and returns
// the windows used since the previous call in *used. Synchronous.
cudaError_t fy_noise_test_paths(int force_radix, int* used) {
    int u = 0, zero = 0;
    cudaError_t e = cudaMemcpyFromSymbol(&u, noise_window_used, sizeof u);
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(noise_window_used, &zero, sizeof zero);
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(noise_force_radix, &force_radix, sizeof force_radix);
    if (e == cudaSuccess && used) *used = u;
    return e;
}

// Bounded waits of this unit's box passes that expired (see fy_zbox.cuh); 0 expected.
int fy_noise_wait_timeouts() { return fyzb::timeouts(); }
cudaError_t fy_noise_set_first_wait_polls(int polls) { return fyzb::set_first_wait_polls(polls); }
