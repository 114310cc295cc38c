// FP64 quotients for GB300, whose FP64 pipe issues at 1/64 of the FP32 rate: a
// division is some ten FP64 instructions.  Source of its own so that a host
// program can compile it and compare with the division.
#pragma once

namespace fipi {

// a / b with r = 1/b rounded to nearest at hand: the quotient estimate corrected
// by its exact remainder is the correctly rounded quotient (P. Markstein, IBM J.
// Res. Dev. 34, 1990), so the results are those of the division, in three
// FP64 instructions instead of about ten.  Infinite, NaN and extreme values
// take the division: quotients outside 2^-512 to 2^512, and numerators below 2^-959,
// whose remainder would lose bits below the subnormals.  |b| < 2^1000.
__device__ __forceinline__ double div_by(double a, double b, double r) {
    const double q = a * r;
    const int e = (__double2hiint(q) >> 20) & 0x7ff, ea = (__double2hiint(a) >> 20) & 0x7ff;
    if ((unsigned)(e - 511) > 1024u || ea < 64) return (__double_as_longlong(a) << 1) == 0 ? q : a / b;
    return fma(fma(-q, b, a), r, q);
}

// 1/x as an unevaluated sum hi + lo, to about 104 bits.
struct Recip {
    double hi, lo;
};
// From an FP32 estimate r (converted both ways on the bits; a conversion or a
// division runs on the FP64 pipe) one third-order step r (1 + e + e^2),
// e = 1 - x r, |e| < 2^-20, gives hi; the remainder of hi gives lo: five FP64
// instructions.  x outside (2^-126, 2^126), negative or NaN: the division.
__device__ __forceinline__ Recip recip(double x) {
    Recip o;
    const int h = __double2hiint(x);
    if ((unsigned)(h - ((1023 - 126) << 20)) >= (252u << 20)) {
        o.hi = 1.0 / x;
        o.lo = fma(-x, o.hi, 1.0) * o.hi;
        if (!(fabs(o.lo) < fabs(o.hi))) o.lo = 0.0;  // 0, infinity, NaN
        return o;
    }
    const float r0 = __fdividef(1.f, __int_as_float(((h - (896 << 20)) << 3) | (int)((unsigned)__double2loint(x) >> 29)));
    const int b = __float_as_int(r0);
    const double r = __hiloint2double((b >> 3) + (896 << 20), b << 29);
    const double e = fma(-x, r, 1.0);
    o.hi = fma(r, fma(e, e, e), r);
    o.lo = fma(-x, o.hi, 1.0) * o.hi;
    return o;
}
// a / x, two FP64 instructions: a lo carries a relative error of 2^-53 on at
// most 2^-52 of the quotient, and the sum is rounded once, so the result is
// the division's unless the quotient lies within 2^-103 of the middle of two
// values.  (Quotients below 2^-960 keep one unit; an infinite a may give NaN.)
__device__ __forceinline__ double over(double a, Recip r) { return fma(a, r.hi, a * r.lo); }

// The projection of one mode (main.cpp:177-178), f - k (k.f)/k^2 over mu k^2, a
// component at a time: s = (k.f)/k^2, r = 1/(mu k^2).  Three roundings, a fused
// multiply-add among them, where the reference's order has four.
__device__ __forceinline__ double projected(double f, double k, double s, Recip r) { return over(fma(-k, s, f), r); }

// Density at phase c, (1 + c)/2 rho1 + (1 - c)/2 rho2 (main.cpp:149-172), from the
// halved densities, which round as the reference's order does (halving is
// exact) in four FP64 instructions a point instead of six.  (c times half
// the difference plus half the sum, one instruction, has errors up to 1.5 times as large.)
template <typename T> __device__ __forceinline__ T mean_density(T c, T half1, T half2) {
    return (c + T(1)) * half1 + (T(1) - c) * half2;
}

// Terms of one contact pair at distance |d| < r_eq in the adjoint of the contact
// forces, F(d) = (r_eq - |d|) ramp k_n d / |d|: dF^T dl into lam, F . li / k_n into kn.
// Quotients and products are the ones of
//   a = r_eq / |d| - 1,  b = r_eq / |d|^3 (d . dl),  lam += ramp k_n (a dl - b d),
//   kn += (r_eq - |d|) ramp / |d| (d . li).
// (To be compiled without contraction.)
__device__ __forceinline__ void pair_adjoint(const double d[3], double r_eq, double rmp, double k_n,
                                             const double dl[3], const double li[3], double lam[3], double& kn) {
    const double dn = sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
    // 0 < dn < r_eq on the bits (false for NaN)
    const unsigned long long bits = (unsigned long long)__double_as_longlong(dn);
    if (bits == 0ull || bits >= (unsigned long long)__double_as_longlong(r_eq)) return;
    const double sc = rmp * k_n;
    const Recip r1 = recip(dn), r3 = recip(dn * dn * dn);
    const double a = over(r_eq, r1) - 1.0;
    const double b = over(r_eq, r3) * (d[0] * dl[0] + d[1] * dl[1] + d[2] * dl[2]);
    for (int e = 0; e < 3; ++e) lam[e] += sc * (a * dl[e] - b * d[e]);
    kn += over((r_eq - dn) * rmp, r1) * (d[0] * li[0] + d[1] * li[1] + d[2] * li[2]);
}

}  // namespace fipi
