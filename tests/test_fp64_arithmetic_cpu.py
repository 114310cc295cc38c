"""The FP64 quotients of csrc/fp64.cuh, compiled for the host, against the
division they stand for."""
import subprocess
from pathlib import Path

import pytest

REPO = Path(__file__).resolve().parent.parent

# CUDA's names for the host.  The FP32 reciprocal estimate is off by up to the
# two units its documentation allows.
HOST = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>
#define __device__
#define __forceinline__ inline
using std::fabs; using std::fma;
static std::mt19937_64 rng(7);
template <class A, class B> static A bits(B b) { A a; std::memcpy(&a, &b, sizeof a); return a; }
static int __double2hiint(double x) { return (int)(bits<uint64_t>(x) >> 32); }
static int __double2loint(double x) { return (int)(uint32_t)bits<uint64_t>(x); }
static double __hiloint2double(int h, int l) { return bits<double>(((uint64_t)(uint32_t)h << 32) | (uint32_t)l); }
static long long __double_as_longlong(double x) { return bits<long long>(x); }
static float __int_as_float(int i) { return bits<float>(i); }
static int __float_as_int(float f) { return bits<int>(f); }
static float __fdividef(float a, float b) { return __int_as_float(__float_as_int(a / b) + (int)(rng() % 5) - 2); }
#include "fp64.cuh"
using namespace fipi;
// random mantissa and sign, exponent in [lo, hi)
static double draw(int lo, int hi) {
    const uint64_t m = rng();
    return std::ldexp(1.0 + (double)(m >> 12) * 0x1p-52, lo + (int)(rng() % (uint64_t)(hi - lo))) * (m & 1 ? -1 : 1);
}
"""

OVER = r"""
int main() {
    long bad = 0;
    const int ranges[][4] = {{-60, 20, 1, 40}, {-300, 300, -125, 126}, {-400, 400, -200, 300}};
    for (auto& r : ranges)
        for (long i = 0; i < 4000000; ++i) {
            const double a = draw(r[0], r[1]), x = fabs(draw(r[2], r[3]));
            bad += over(a, recip(x)) != a / x;
        }
    for (double a : {0.0, 1.0, -3.5})
        for (double x : {3.0, 0x1p-126, 0x1p126, 0x1p-1022, (double)INFINITY}) bad += over(a, recip(x)) != a / x;
    bad += over(1.0, recip(0.0)) != INFINITY || !std::isnan(over(0.0, recip(0.0))) || !std::isnan(over(1.0, recip(NAN)));
    std::printf("%ld\n", bad);
    return bad != 0;
}
"""

DIV_BY = r"""
int main() {
    long bad = 0;
    const int ranges[][4] = {{-60, 60, -40, 40}, {-1074, 1000, -1000, 999}, {-1074, -900, -1000, -400}};
    for (auto& r : ranges)
        for (long i = 0; i < 4000000; ++i) {
            const double a = draw(r[0], r[1]), b = draw(r[2], r[3]);
            bad += bits<uint64_t>(div_by(a, b, 1.0 / b)) != bits<uint64_t>(a / b);
        }
    for (double a : {0.0, -0.0, 1.0, (double)INFINITY, (double)NAN})
        for (double b : {3.0, -3.0, 0.0, (double)INFINITY, (double)NAN}) {
            const double x = div_by(a, b, 1.0 / b), y = a / b;
            bad += std::isnan(y) ? !std::isnan(x) : x != y || std::signbit(x) != std::signbit(y);
        }
    std::printf("%ld\n", bad);
    return bad != 0;
}
"""

# relative errors of the projection against extended precision: no larger than the
# reference's expression (main.cpp:177-178), for modes that are nearly
# divergence-free, nearly along k and neither
PROJECT = r"""
int main() {
    int bad = 0;
    for (double along : {1e-6, 1.0, 1e3}) {
        double here2 = 0, ref2 = 0, here_max = 0, ref_max = 0;
        for (int i = 0; i < 1000000; ++i) {
            const double k[3] = {draw(-6, 3), draw(-6, 3), draw(-6, 3)}, mu = fabs(draw(-10, 4));
            double f[3] = {draw(-8, 0), draw(-8, 0), draw(-8, 0)};
            const double k2 = k[0] * k[0] + k[1] * k[1] + k[2] * k[2], mk2 = mu * k2;
            const double c = (1 - along) * (k[0] * f[0] + k[1] * f[1] + k[2] * f[2]) / k2;
            for (int d = 0; d < 3; ++d) f[d] -= c * k[d];
            const double dot = k[0] * f[0] + k[1] * f[1] + k[2] * f[2];
            const Recip r = recip(mk2);
            const double s = over(dot, recip(k2));
            long double u2 = 0, eh = 0, er = 0;
            for (int d = 0; d < 3; ++d) {
                const long double u = ((long double)f[d] - (long double)k[d] * dot / k2) / mk2;
                const long double h = projected(f[d], k[d], s, r) - u, g = (f[d] - (k[d] * dot) / k2) / mk2 - u;
                u2 += u * u; eh += h * h; er += g * g;
            }
            here2 += (double)(eh / u2); ref2 += (double)(er / u2);
            here_max = std::fmax(here_max, (double)(eh / u2)); ref_max = std::fmax(ref_max, (double)(er / u2));
        }
        std::printf("%g: rms %.4g against %.4g, max %.4g against %.4g\n", along, std::sqrt(here2 / 1e6), std::sqrt(ref2 / 1e6),
                    std::sqrt(here_max), std::sqrt(ref_max));
        // where both round alike the sums differ by their sampling: 3 / sqrt(2e6) of the mean square
        const double more = 1 + 3 / std::sqrt(2e6);
        bad |= here2 > more * ref2 || here_max > more * ref_max;
    }
    return bad;
}
"""


def _run(tmp_path, body):
    src, exe = tmp_path / "h.cpp", tmp_path / "h"
    src.write_text(HOST + body)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", str(REPO / "fipi_gb300/csrc"), str(src),
                    "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
    return r.stdout


@pytest.mark.parametrize("body", [OVER, DIV_BY], ids=["over", "div_by"])
def test_quotients_are_the_divisions(tmp_path, body):
    _run(tmp_path, body)


def test_projection_is_as_accurate_as_the_reference(tmp_path):
    _run(tmp_path, PROJECT)


# the buoyancy's density: the reference's expression bit for bit
DENSITY = r"""
int main() {
    long bad = 0;
    const double rho[][2] = {{1e-3, 1e-3}, {1e-3, 5e-2}, {1.0, 1e-3}, {2.0, 1.0}, {0.7, 0.3}, {1e3, 1.2}, {1.0, 0.0}};
    for (auto& r : rho)
        for (int i = 0; i < 1000000; ++i) {
            const double c = i % 2 ? 1.1 * ((double)(rng() >> 11) * 0x1p-52 - 1.0) : draw(-60, 2);
            bad += mean_density(c, r[0] * 0.5, r[1] * 0.5) != ((c + 1.0) / 2.0) * r[0] + ((c * -1.0 + 1.0) / 2.0) * r[1];
            const float f = (float)c, r0 = (float)r[0], r1 = (float)r[1];
            bad += mean_density(f, r0 * 0.5f, r1 * 0.5f) != ((f + 1.f) / 2.f) * r0 + ((f * -1.f + 1.f) / 2.f) * r1;
        }
    std::printf("%ld\n", bad);
    return bad != 0;
}
"""


def test_density_is_the_references(tmp_path):
    _run(tmp_path, DENSITY)


# the adjoint's pair terms: the sums of the expressions with divisions, bit for bit,
# from nearly touching centres to the contact range, and nothing outside it
PAIR = r"""
int main() {
    long bad = 0;
    for (int i = 0; i < 4000000; ++i) {
        const double r_eq = fabs(draw(-4, 6)), rmp = (double)(1 + rng() % 100) / 100, k_n = fabs(draw(-6, 6));
        double d[3] = {draw(-20, 0), draw(-20, 0), draw(-20, 0)}, dl[3], li[3];
        const double far = r_eq * std::pow(2.0, -(double)(rng() % 4096) / 128 + 0.1) /
                           std::sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
        for (int e = 0; e < 3; ++e) { d[e] *= far; dl[e] = draw(-10, 3); li[e] = draw(-10, 3); }
        if (i % 1000 == 0) d[0] = d[1] = d[2] = 0.0;
        if (i % 1000 == 1) d[i % 3] = NAN;
        double lam[3] = {draw(-5, 5), draw(-5, 5), draw(-5, 5)}, kn = draw(-5, 5);
        double want[3] = {lam[0], lam[1], lam[2]}, want_kn = kn;
        const double dn = std::sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
        if (dn < r_eq && dn != 0.0) {
            const double a = r_eq / dn - 1.0, b = r_eq / (dn * dn * dn) * (d[0] * dl[0] + d[1] * dl[1] + d[2] * dl[2]);
            for (int e = 0; e < 3; ++e) want[e] += rmp * k_n * (a * dl[e] - b * d[e]);
            want_kn += (r_eq - dn) * rmp / dn * (d[0] * li[0] + d[1] * li[1] + d[2] * li[2]);
        }
        pair_adjoint(d, r_eq, rmp, k_n, dl, li, lam, kn);
        bad += lam[0] != want[0] || lam[1] != want[1] || lam[2] != want[2] || kn != want_kn;
    }
    std::printf("%ld\n", bad);
    return bad != 0;
}
"""


def test_pair_adjoint_is_the_divisions(tmp_path):
    _run(tmp_path, PAIR)
