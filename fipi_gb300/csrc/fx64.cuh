// Block fixed-point arithmetic of the FP64 form's transforms (sm_103a).
//
// GB300 issues FP64 at 1/64 of its FP32 rate (2 lanes per clock and SM,
// measured 0.53 T instructions/s) but 64-bit integer additions at 58 and
// 32 x 32 + 64-bit multiply-adds at 24 lanes per clock.  A radix-8 stage with
// its twiddles is about 80 FP64 instructions for 8 values; in integers it ran
// at 508 G values/s against 53 G.  So a row is converted to integers with
// one exponent for the row, transformed in integers, and converted back:
//
//   value = integer * 2^(E - 1022 - B),   E = largest exponent field of the row
//
// puts the largest component in [2^(B-1), 2^B).  Twiddled stages divide by four
// (the products' natural scale) and round to nearest at the last bit.  B is
// the larger of two bounds that keep every intermediate below 2^63:
//  - any row of N <= 512 grows by at most 32 (N = 512) or 16 in modulus on its
//    way: B = 57 or 58, four bits and more below an FP64 of the row's largest
//    value;
//  - no intermediate exceeds the row's sum of moduli, so a row with few large
//    values (a spectrum with a dominant mode) may start with that sum < 2^62.
// An FP64 transform rounds at the level of the row's norm as well.  Relative
// L2 errors of 3-D transforms (64^3, 128 x 128 x 64, and 16- to 512-point axes;
// uniform noise, offset noise, an interface, a spike, one mode; both
// directions) against extended precision: 0.2 to 0.95 of the FP64 codelets'
// (uniform noise 2.7e-16 -> 0.9e-16; offset noise, inverse, 512-point rows
// 1.75e-16 -> 1.3e-16; with the growth bound alone 6.8e-16).
// Measured at 256^3: three-field Y pass 1207 -> 276 us, force pass 4250 -> 1001,
// projection round trip 4510 -> 1209 (with the warp-owned rows and columns and the
// quotients of fp64.cuh).
//
// Rows with an infinity or a NaN (E = 0x7ff) come out as NaN throughout.
// Rows below 2^-959 are scaled up by 2^200 first, so subnormal inputs
// enter with all their bits; results are representable up to the largest FP64
// value and down to its subnormals (fx_unrow).
#pragma once

#include <type_traits>

#include "common.cuh"

namespace fipi {

struct fx64 {};  // arithmetic type tag of the transform codelets
template <> struct cplx_of<fx64> { using type = longlong2; };
template <typename C> constexpr bool is_fx = std::is_same<C, longlong2>::value;

__device__ __forceinline__ long long fx_mad(int a, int b, long long c) {
    long long d;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
    return d;
}
__device__ __forceinline__ int fx_lo(long long a) { return (int)(unsigned)(unsigned long long)a; }
__device__ __forceinline__ int fx_hi(long long a) { return (int)(a >> 32); }
// high word of a = hi 2^32 + lo with lo signed
__device__ __forceinline__ int fx_hib(long long a) { return fx_hi(a) + (int)((unsigned)(unsigned long long)a >> 31); }

// Twiddle factors are stored as 2^62 w split into a signed high and a signed
// low word (fx_pack).
inline long long fx_pack(long long w62) {
    const long long hi = (w62 + (1ll << 31)) >> 32;
    const int lo = (int)(w62 - hi * (1ll << 32));
    return (long long)(((unsigned long long)hi << 32) | (unsigned)lo);
}

// a w / 4, or a conj(w) / 4 for the inverse direction.  With a = x1 2^32 +
// x0 and w likewise, the products of two low words are left out (below one
// unit); the middle sum carries half a unit for rounding.
template <int DIR> __device__ __forceinline__ longlong2 fx_mulw(longlong2 a, longlong2 w) {
    const int r1 = fx_hi(w.x), r0 = fx_lo(w.x);
    const int j1 = fx_hi(w.y), j0 = fx_lo(w.y);
    const int i1 = DIR < 0 ? j1 : -j1, i0 = DIR < 0 ? j0 : -j0;  // im part of the factor
    const int n1 = DIR < 0 ? -j1 : j1, n0 = DIR < 0 ? -j0 : j0;  // and its negative
    const int x1 = fx_hib(a.x), x0 = fx_lo(a.x), y1 = fx_hib(a.y), y0 = fx_lo(a.y);
    long long mr = fx_mad(x1, r0, 1ll << 31), mi = fx_mad(x1, i0, 1ll << 31);
    mr = fx_mad(x0, r1, mr);
    mi = fx_mad(x0, i1, mi);
    mr = fx_mad(y1, n0, mr);
    mi = fx_mad(y1, r0, mi);
    mr = fx_mad(y0, n1, mr);
    mi = fx_mad(y0, r1, mi);
    longlong2 o;
    o.x = fx_mad(y1, n1, fx_mad(x1, r1, (long long)fx_hi(mr)));
    o.y = fx_mad(y1, r1, fx_mad(x1, i1, (long long)fx_hi(mi)));
    return o;
}
// a sqrt(1/2) = a + a (sqrt(1/2) - 1)
__device__ __forceinline__ long long fx_rsqrt2(long long a) {
    constexpr long long c = -5402926248376769404ll;  // 2^64 (sqrt(1/2) - 1)
    constexpr int c1 = (int)((c + (1ll << 31)) >> 32);
    constexpr int c0 = (int)(c - (long long)c1 * (1ll << 32));
    const int a1 = fx_hib(a), a0 = fx_lo(a);
    const long long m = fx_mad(a0, c1, fx_mad(a1, c0, 1ll << 31));
    return fx_mad(a1, c1, a) + (long long)fx_hi(m);
}
// a exp(DIR 2 pi i e / 16) for the odd eighths of a turn, e = 2, 6, 10, 14
template <int DIR, int E16> __device__ __forceinline__ longlong2 fx_rot8(longlong2 a) {
    static_assert(E16 % 4 == 2, "an odd eighth of a turn");
    constexpr int q = (DIR < 0 ? 16 - E16 : E16) & 15;  // counter-clockwise sixteenths
    // (x + i y)(c + i s) with |c| = |s| = sqrt(1/2)
    constexpr bool cneg = q == 6 || q == 10, sneg = q == 10 || q == 14;
    const long long xr = cneg ? -a.x : a.x, yr = cneg ? -a.y : a.y;
    longlong2 o;
    o.x = fx_rsqrt2(sneg ? xr + a.y : xr - a.y);
    o.y = fx_rsqrt2(sneg ? yr - a.x : yr + a.x);
    return o;
}
__device__ __forceinline__ longlong2 fx_quarter(longlong2 a) {
    longlong2 o;
    o.x = (a.x + 2) >> 2;
    o.y = (a.y + 2) >> 2;
    return o;
}

// Size of a row: mag, the upper word of its largest |component| (ordered like
// it), and l1, the sum of max(|re|, |im|) in FP32 (used for rows well inside
// the FP32 range only): the moduli sum to at most sqrt(2) l1.
struct FxSize {
    int mag = 0;
    float l1 = 0.f;
    __device__ __forceinline__ void add(double2 v) {
        const int h = max(__double2hiint(v.x) & 0x7fffffff, __double2hiint(v.y) & 0x7fffffff);
        mag = max(mag, h);
        // as FP32 from the upper word (the FP32 exponent field is 896 less);
        // a conversion instruction would run on the FP64 pipe
        l1 += __int_as_float(max(h - (896 << 20), 0) << 3);
    }
};

struct FxSlot {  // FxSize in shared memory
    int mag;
    float l1;
};

// x 2^(1022 + B - E) rounded towards zero, for rows whose largest exponent
// field is E >= 64 (smaller ones: fx_row).
__device__ __forceinline__ long long fx_from(double x, int E, int B) {
    const int hi = __double2hiint(x);
    const int s = min(E + 63 - B - ((hi >> 20) & 0x7ff), 63);
    const unsigned long long m =
        (((unsigned long long)(unsigned)((hi & 0xfffff) | 0x100000) << 32) | (unsigned)__double2loint(x)) << 10;
    const long long r = (long long)(m >> s);
    return hi < 0 ? -r : r;
}
// a 2^q, rounded to nearest (the rounding carry runs into the exponent field),
// for -1022 <= q <= 960, where every result but zero is a normal number.
__device__ __forceinline__ double fx_to(long long a, int q) {
    const int sg = fx_hi(a) & 0x80000000;
    const unsigned long long u = a < 0 ? 0ull - (unsigned long long)a : (unsigned long long)a;
    const int z = __clzll((long long)u);  // >= 1: |a| < 2^63
    const unsigned long long r = ((u << (z - 1)) + 0x200ull) >> 10;  // leading one at bit 52
    const int e = q + 1085 - z;  // exponent field less one (1023 + 63)
    return u == 0 ? 0.0 : __hiloint2double(((int)(r >> 32) + (e << 20)) | sg, (int)(unsigned)r);
}
// The same by the FP64 pipe's conversion instruction and an exponent addition:
// one FP64 instruction instead of a dozen integer ones.
__device__ __forceinline__ double fx_to_cvt(long long a, int q) {
    const double d = __ll2double_rn(a);
    return a == 0 ? 0.0 : __hiloint2double(__double2hiint(d) + (q << 20), __double2loint(d));
}
// One component on either pipe: 1099 G conversions/s against 844 (integer)
// and 593 (FP64 pipe), measured alone.
__device__ __forceinline__ double2 fx_to(longlong2 a, int q) {
    double2 o;
    o.x = fx_to(a.x, q);
    o.y = fx_to_cvt(a.y, q);
    return o;
}

// A row of K values per thread into integers.  BITS: the growth bound's B;
// L1: log2 of the bound on the row's sum of magnitudes.  Returns E and the
// exponent q of the integers' unit.
struct FxExp {
    int E, q;
};
template <int K, int BITS, int L1> __device__ __forceinline__ FxExp fx_row(double2* v, FxSize z, longlong2* o) {
    int E = z.mag >> 20, back = 0, B = BITS;
    if (E < 64) {  // subnormal or tiny: 2^200 larger (exact)
#pragma unroll
        for (int i = 0; i < K; ++i) {
            v[i].x *= 0x1p200;
            v[i].y *= 0x1p200;
        }
        E = max(E, 1) + 200;
        back = 200;
    }
    if ((unsigned)(E - (1023 - 90)) < 180u) {
        // the moduli sum to less than 2^(e - 126), e the exponent field of
        // sqrt(2) l1 (with a margin for the FP32 sums and the cut-off words)
        const int e = __float_as_int(z.l1 * 1.4157f) >> 23;
        B = max(B, L1 - (e - 126) + (E - 1022));
    }
#pragma unroll
    for (int i = 0; i < K; ++i) {
        o[i].x = fx_from(v[i].x, E, B);
        o[i].y = fx_from(v[i].y, E, B);
    }
    return {E, E - 1022 - B - back};
}
// Integers of such a row back to FP64, times 2^shift.
template <int K> __device__ __forceinline__ void fx_unrow(const longlong2* o, FxExp x, int shift, double2* v) {
    // rows whose values may leave the normal range: converted inside it, then
    // scaled by a power of two, which rounds subnormals and overflows as FP64 does
    const int q = x.q + shift, adj = q < -1022 ? 400 : q > 960 ? -200 : 0;
#pragma unroll
    for (int i = 0; i < K; ++i) v[i] = fx_to(o[i], q + adj);
    if (adj != 0) {
        const double f = adj > 0 ? 0x1p-400 : 0x1p200;
#pragma unroll
        for (int i = 0; i < K; ++i) {
            v[i].x *= f;
            v[i].y *= f;
        }
    }
    if (x.E == 0x7ff) {
#pragma unroll
        for (int i = 0; i < K; ++i) v[i].x = v[i].y = __hiloint2double(0x7ff80000, 0);
    }
}

// Size of a row over its Tn threads, which lie within one warp (Tn a power of
// two; every lane of the warp calls).
template <int Tn> __device__ __forceinline__ FxSize fx_row_size(FxSize z) {
#pragma unroll
    for (int o = 1; o < Tn && o < 32; o <<= 1) {
        z.mag = max(z.mag, __shfl_xor_sync(0xffffffffu, z.mag, o));
        z.l1 += __shfl_xor_sync(0xffffffffu, z.l1, o);
    }
    return z;
}
// Size of each of the TZ columns of a block of NT threads, column =
// thread % TZ (TZ a power of two).  `slot`: (NT + 31) / 32 * TZ entries; the
// block synchronises once, and a slot array may be used again after the next
// block barrier.
template <int TZ, int NT> __device__ __forceinline__ FxSize fx_column_size(FxSize z, FxSlot* slot) {
    constexpr int NW = (NT + 31) / 32;
    constexpr int W = NT < 32 ? NT : 32;  // lanes of a warp
    constexpr unsigned mask = W == 32 ? 0xffffffffu : (1u << (W & 31)) - 1u;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = TZ; o < W; o <<= 1) {
        z.mag = max(z.mag, __shfl_xor_sync(mask, z.mag, o));
        z.l1 += __shfl_xor_sync(mask, z.l1, o);
    }
    if (lane < TZ) slot[w * TZ + lane] = FxSlot{z.mag, z.l1};
    __syncthreads();
    z = FxSize{};
#pragma unroll
    for (int k = 0; k < NW; ++k) {
        const FxSlot y = slot[k * TZ + lane % TZ];
        z.mag = max(z.mag, y.mag);
        z.l1 += y.l1;
    }
    return z;
}

}  // namespace fipi
