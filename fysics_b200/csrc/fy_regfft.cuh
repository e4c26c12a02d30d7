// fy_regfft.cuh -- line transforms that stay in registers, with one exchange.
//
// The Stockham transform of fy_fft.cuh with the points divided differently. There a thread holds
// E = 16 or 24 points and every radix pass crosses shared memory between two CTA barriers; here it
// holds E points, so that the first TWO passes of a line -- the head, PA = 4*4, 8*4 or 3*8 points
// -- run inside the thread's registers, with twiddles that are compile-time constants, the line
// crosses shared memory ONCE, and the remaining passes -- the tail -- run in registers again:
//   n      64      128      256      512    |    96       192      384
//   passes 4,4|4   4,4|8    8,4|8    8,4|8,2|    3,8|4    3,8|8    3,8|8,2
//   E      16      16       32       32     |    24       24       48
//   TPL    4       8        8        16     |    4        8        8      threads per line
// (64 and 128 with E = 32 leave a 128^3 volume 7 warps an SM: its chain 309 us, 303 with 16.)
// A point costs 38 thread instructions a transform (about 50 before). Heads of 64 points (E = 64,
// 8*8) were tried too: 35 instructions, but only 12 warps fit an SM and latency ruled (256^3
// passes 1.5 to 2.8 times slower than with E = 32).
// Ownership: before the head and after the tail thread t of a line holds the points t + TPL*m at
// v[m] (natural slots), so an inverse transform continues a forward one without an exchange; a
// caller reads its inputs and writes its outputs at those points. After the head the thread holds
// whole blocks of PA points, (t + TPL*b)*PA + q.
// Why in-thread heads close: pass 1 (radix R1) needs points N/R1 apart. Pass 0 turns the points
// t + TPL*b (+ r*N/R0) into (t + TPL*b)*R0 + r, and N/R1 = TPL*R0*(E/PA): the partners are the
// same thread's other b.
#pragma once
#include "fy_fft.cuh"

namespace rf {

// Axis lengths with a register plan. 768 and 1024 would need a tail of three passes or twice the
// threads and shared memory a tile; they stay on fy_fft.cuh.
constexpr bool served(int n) {
    return n == 64 || n == 96 || n == 128 || n == 192 || n == 256 || n == 384 || n == 512;
}
constexpr int elems(int n) { return n % 3 ? (n <= 128 ? 16 : 32) : (n == 384 ? 48 : 24); }
constexpr int head_len(int n) { return n % 3 ? (n <= 128 ? 16 : 32) : 24; }
constexpr int head_r0(int n) { return n % 3 ? (n <= 128 ? 4 : 8) : 3; }
constexpr int head_r1(int n) { return n % 3 ? 4 : 8; }
constexpr int tpl(int n) { return n / elems(n); }

// exp(2*pi*i*m/32) and exp(2*pi*i*m/24), FP64 rounded once to float like the twiddle tables.
template <int PA> constexpr float root_c(int m) {
    constexpr float c32[32] = {
        0x1.0000000000000p+0f, 0x1.f6297c0000000p-1f, 0x1.d906bc0000000p-1f, 0x1.a9b6620000000p-1f, 0x1.6a09e60000000p-1f,
        0x1.1c73b40000000p-1f, 0x1.87de2a0000000p-2f, 0x1.8f8b840000000p-3f, 0x1.1a62640000000p-54f, -0x1.8f8b840000000p-3f,
        -0x1.87de2a0000000p-2f, -0x1.1c73b40000000p-1f, -0x1.6a09e60000000p-1f, -0x1.a9b6620000000p-1f, -0x1.d906bc0000000p-1f,
        -0x1.f6297c0000000p-1f, -0x1.0000000000000p+0f, -0x1.f6297c0000000p-1f, -0x1.d906bc0000000p-1f, -0x1.a9b6620000000p-1f,
        -0x1.6a09e60000000p-1f, -0x1.1c73b40000000p-1f, -0x1.87de2a0000000p-2f, -0x1.8f8b840000000p-3f, -0x1.a793940000000p-53f,
        0x1.8f8b840000000p-3f, 0x1.87de2a0000000p-2f, 0x1.1c73b40000000p-1f, 0x1.6a09e60000000p-1f, 0x1.a9b6620000000p-1f,
        0x1.d906bc0000000p-1f, 0x1.f6297c0000000p-1f};
    constexpr float c24[24] = {
        0x1.0000000000000p+0f, 0x1.ee8dd40000000p-1f, 0x1.bb67ae0000000p-1f, 0x1.6a09e60000000p-1f, 0x1.0000000000000p-1f,
        0x1.0907dc0000000p-2f, 0x1.1a62640000000p-54f, -0x1.0907dc0000000p-2f, -0x1.0000000000000p-1f, -0x1.6a09e60000000p-1f,
        -0x1.bb67ae0000000p-1f, -0x1.ee8dd40000000p-1f, -0x1.0000000000000p+0f, -0x1.ee8dd40000000p-1f, -0x1.bb67ae0000000p-1f,
        -0x1.6a09e60000000p-1f, -0x1.0000000000000p-1f, -0x1.0907dc0000000p-2f, -0x1.a793940000000p-53f, 0x1.0907dc0000000p-2f,
        0x1.0000000000000p-1f, 0x1.6a09e60000000p-1f, 0x1.bb67ae0000000p-1f, 0x1.ee8dd40000000p-1f};
    return PA == 24 ? c24[m % 24] : c32[m * (32 / PA) & 31];
}
template <int PA> constexpr float root_s(int m) {
    constexpr float s32[32] = {
        0x0.0p+0f, 0x1.8f8b840000000p-3f, 0x1.87de2a0000000p-2f, 0x1.1c73b40000000p-1f, 0x1.6a09e60000000p-1f,
        0x1.a9b6620000000p-1f, 0x1.d906bc0000000p-1f, 0x1.f6297c0000000p-1f, 0x1.0000000000000p+0f, 0x1.f6297c0000000p-1f,
        0x1.d906bc0000000p-1f, 0x1.a9b6620000000p-1f, 0x1.6a09e60000000p-1f, 0x1.1c73b40000000p-1f, 0x1.87de2a0000000p-2f,
        0x1.8f8b840000000p-3f, 0x1.1a62640000000p-53f, -0x1.8f8b840000000p-3f, -0x1.87de2a0000000p-2f, -0x1.1c73b40000000p-1f,
        -0x1.6a09e60000000p-1f, -0x1.a9b6620000000p-1f, -0x1.d906bc0000000p-1f, -0x1.f6297c0000000p-1f, -0x1.0000000000000p+0f,
        -0x1.f6297c0000000p-1f, -0x1.d906bc0000000p-1f, -0x1.a9b6620000000p-1f, -0x1.6a09e60000000p-1f, -0x1.1c73b40000000p-1f,
        -0x1.87de2a0000000p-2f, -0x1.8f8b840000000p-3f};
    constexpr float s24[24] = {
        0x0.0p+0f, 0x1.0907dc0000000p-2f, 0x1.0000000000000p-1f, 0x1.6a09e60000000p-1f, 0x1.bb67ae0000000p-1f,
        0x1.ee8dd40000000p-1f, 0x1.0000000000000p+0f, 0x1.ee8dd40000000p-1f, 0x1.bb67ae0000000p-1f, 0x1.6a09e60000000p-1f,
        0x1.0000000000000p-1f, 0x1.0907dc0000000p-2f, 0x1.1a62640000000p-53f, -0x1.0907dc0000000p-2f, -0x1.0000000000000p-1f,
        -0x1.6a09e60000000p-1f, -0x1.bb67ae0000000p-1f, -0x1.ee8dd40000000p-1f, -0x1.0000000000000p+0f, -0x1.ee8dd40000000p-1f,
        -0x1.bb67ae0000000p-1f, -0x1.6a09e60000000p-1f, -0x1.0000000000000p-1f, -0x1.0907dc0000000p-2f};
    return PA == 24 ? s24[m % 24] : s32[m * (32 / PA) & 31];
}

// f(integral_constant<I>) for I = B .. E-1
template <int B, int E, class F>
FY_D void sfor(F&& f) {
    if constexpr (B < E) {
        f(std::integral_constant<int, B>{});
        sfor<B + 1, E>(f);
    }
}

// The two head passes. Slot (b + rp*B1) + r*G0 ends with output q = r + rp*R0 of block b.
template <int N, int SIGN>
FY_D void head(float2 (&v)[elems(N)]) {
    constexpr int E = elems(N), PA = head_len(N), R0 = head_r0(N), R1 = head_r1(N), G0 = E / R0, B1 = G0 / R1;
#pragma unroll
    for (int b = 0; b < G0; ++b) {
        float2 u[R0];
#pragma unroll
        for (int r = 0; r < R0; ++r) u[r] = v[b + r * G0];
        Bfly<R0>::run(u, (float)SIGN);
#pragma unroll
        for (int r = 0; r < R0; ++r) v[b + r * G0] = u[r];
    }
    sfor<0, B1>([&](auto bc) {
        sfor<0, R0>([&](auto rc) {
            constexpr int b = decltype(bc)::value, r = decltype(rc)::value;
            float2 u[R1];
            sfor<0, R1>([&](auto pc) {
                constexpr int rp = decltype(pc)::value;
                u[rp] = v[(b + rp * B1) + r * G0];
                if constexpr (r * rp != 0) {
                    constexpr float c = root_c<PA>(r * rp), s = SIGN < 0 ? -root_s<PA>(r * rp) : root_s<PA>(r * rp);
                    u[rp] = cmul(u[rp], make_float2(c, s));
                }
            });
            Bfly<R1>::run(u, (float)SIGN);
            sfor<0, R1>([&](auto pc) { constexpr int rp = decltype(pc)::value; v[(b + rp * B1) + r * G0] = u[rp]; });
        });
    });
}

// After the head: st(block, q, value) for the thread's blocks b (block index t + TPL*b) and
// their points q.
template <int N, class ST>
FY_D void head_store(const float2 (&v)[elems(N)], int t, ST st) {
    constexpr int E = elems(N), R0 = head_r0(N), R1 = head_r1(N), G0 = E / R0, B1 = G0 / R1, TPL = tpl(N);
#pragma unroll
    for (int b = 0; b < B1; ++b)
#pragma unroll
        for (int r = 0; r < R0; ++r)
#pragma unroll
            for (int rp = 0; rp < R1; ++rp) st(t + TPL * b, r + rp * R0, v[(b + rp * B1) + r * G0]);
}

// The tail's twiddles, gathered from the length-N table exp(+2*pi*i*m/N) so that the lanes of a
// warp, which differ in k, read consecutive entries: first pass (radix R, span PA) entry
// (r-1)*PA + k = w^(r*k) of order PA*R, then (384, 512) the radix-2 pass's N/2 entries.
template <int N> struct Tail {
    static constexpr int PA = head_len(N), PB = N / PA, R = PB > 8 ? 8 : PB, R2 = PB / R, TWS = N / (PA * R);
    static constexpr int first = (R - 1) * PA, count = first + (R2 > 1 ? N / 2 : 0);
    static_assert(R2 == 1 || R2 == 2, "one more radix-2 pass at most");
};
template <int N>
FY_D void load_tail_twiddles(float2* __restrict__ s, const float2* __restrict__ tw) {
    using T = Tail<N>;
    for (int i = threadIdx.x; i < T::count; i += blockDim.x) {
        const int r = i / T::PA + 1, k = i - (r - 1) * T::PA;
        s[i] = __ldg(tw + (i < T::first ? r * k * T::TWS : i - T::first));
    }
}

// The tail passes on natural slots; the result is in natural slots. stw: the twiddles above.
template <int N, int SIGN>
FY_D void tail(float2 (&v)[elems(N)], int t, const float2* __restrict__ stw) {
    using T = Tail<N>;
    constexpr int E = elems(N), PA = head_len(N), TPL = tpl(N), R = T::R, G = E / R;
#pragma unroll
    for (int b = 0; b < G; ++b) {
        const int k = t + TPL * (b % (PA / TPL));                // (t + TPL*b) mod PA
        float2 u[R];
        u[0] = v[b];
#pragma unroll
        for (int r = 1; r < R; ++r) {
            float2 w = stw[(r - 1) * PA + k];
            if (SIGN < 0) w.y = -w.y;
            u[r] = cmul(v[b + r * G], w);
        }
        Bfly<R>::run(u, (float)SIGN);
#pragma unroll
        for (int r = 0; r < R; ++r) v[b + r * G] = u[r];
    }
    if constexpr (T::R2 > 1) {                                   // one radix-2 pass, span 8*PA = N/2
        constexpr int GB = G / 2;                                // the thread's points of a PA block
        float2 w2[E];
#pragma unroll
        for (int b = 0; b < GB; ++b)
#pragma unroll
            for (int r = 0; r < R; ++r) {
                float2 u[2] = {v[b + r * G], v[b + GB + r * G]};
                float2 w = stw[T::first + t + TPL * b + r * PA]; // butterfly j' of the span
                if (SIGN < 0) w.y = -w.y;
                u[1] = cmul(u[1], w);
                Bfly<2>::run(u, (float)SIGN);
                const int m = b + r * (PA / TPL);                // point j' = t + TPL*m
                w2[m] = u[0];
                w2[m + E / 2] = u[1];                            // + N/2
            }
#pragma unroll
        for (int m = 0; m < E; ++m) v[m] = w2[m];
    }
}

}  // namespace rf
