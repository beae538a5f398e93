"""The shared-reciprocal quotients (lg_quotient.cuh) against the division, on
the CPU: the header's host form with seeds of any error up to 2^-19.
Divisors next to those with every mantissa bit set, which no square has,
dividends next to rounding midpoints and powers of two, quotients near 2,
zeros, and operands out of range, which quotient_suspect and recip_range have
to pick out."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "legendre_b200" / "csrc"

PROGRAM = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>
static std::mt19937_64 rng(7);
static double seed(double c) {  // as coarse as the hardware's, the low word clear
    std::uniform_real_distribution<double> u(-0x1p-19, 0x1p-19);
    if (!std::isnormal(c) || !std::isnormal(1.0 / c)) return std::fabs(c) < 1.0 ? std::copysign(INFINITY, c) : 0.0 * c;
    double y = (1.0 / c) * (1.0 + u(rng));
    uint64_t b;
    std::memcpy(&b, &y, 8);
    b &= 0xffffffff00000000ull;
    std::memcpy(&y, &b, 8);
    return y;
}
#define LG_HOST_RECIP_SEED seed
#include "lg_quotient.cuh"
using namespace lg;
static long checked = 0, wrong = 0, divided = 0;
static bool same(double a, double b) { return (a != a && b != b) || std::memcmp(&a, &b, 8) == 0; }
static void check(bool ok, const char* what, double x, double c) {
    ++checked;
    if (!ok && ++wrong < 10) std::printf("%s: %a / %a\n", what, x, c);
}
static double at(uint64_t mantissa, int e) { return std::ldexp((double)mantissa, e - 52); }
static void quotient(double x, double c) {  // in range
    const double y = recip_rn(c), k = quotient_rn(x, c, y);
    if (low_word(c) == 0xffffffffu) {
        ++divided;
        return;
    }
    check(same(y, 1.0 / c), "reciprocal", 1.0, c);
    check(same(k, x / c), "quotient", x, c);
}
static void guarded(double x, double c) {  // any dividend, c in a mobility's or a face's range
    const double k = quotient_rn(x, c, recip_rn(c)), q = x / c;
    if (low_word(c) == 0xffffffffu) return;
    if (!(c >= 0x1p60) && !(c > 0.0 && c < 0x1p-1021))
        check(quotient_suspect(x, k, 1.0, 1.0) || k == q || (q != q && k != k), "unsuspected", x, c);
    check(quotient_suspect(x, k, 1.0, 1.0) == quotient_suspect(-1.0, 1.0, x, k), "shared test", x, c);
    check(quotient_suspect(x, 1.0, 1.0, 1.0) == (x != 0.0 && std::fabs(x) < kQuotientLow), "low", x, c);
    if (recip_range(c, kQuotientSpan) && std::fabs(x) >= kQuotientLow && std::fabs(x) <= 0x1p100)
        check(same(k, q), "in range", x, c);
    check(!recip_range(c, 0), "no span", x, c);
}
int main() {
    const uint64_t top = (1ull << 53) - 1, one = 1ull << 52;
    for (int k = 0; k < 200; ++k)  // divisors next to a power of two, from below and above
        for (int j = 0; j < 60; ++j)
            for (int e = -3; e <= 3; ++e) {
                quotient(at(one + j, e), at(top - k, e * 5));
                quotient(at(top - j, e), at(top - k, e * 5));
                quotient(at(one, e), at(one + k, j - 30));
            }
    for (int k = 1; k < 400; ++k)  // quotients near 2 next to midpoints, where the first estimate is coarsest
        for (int j = 0; j < 40; ++j) {
            const unsigned __int128 p = (((unsigned __int128)1 << 54) - (2 * j + 1)) * (top - k + 1);
            const uint64_t x = (uint64_t)(p >> 54);
            for (int d = -1; d <= 2; ++d)
                if (x + d >= one && x + d <= top) quotient(at(x + d, 0), at(top - k + 1, 0));
        }
    for (int i = 0; i < 400000; ++i) {  // random and near-midpoint dividends
        const uint64_t c = one | (rng() >> 12) | 1;
        uint64_t inv = c;
        for (int n = 0; n < 6; ++n) inv *= 2 - c * inv;
        const uint64_t m = ((inv * (uint64_t)((int64_t)(rng() % 64) - 32)) & ((1ull << 53) - 1)) | (1ull << 53) | 1;
        unsigned __int128 p = (unsigned __int128)m * c;
        int sh = 0;
        while ((p >> sh) >= ((unsigned __int128)1 << 53)) ++sh;
        const int e = (int)(rng() % 800) - 400;
        quotient(at((uint64_t)(p >> sh), 3), at(c, e));
        quotient(at(one | (rng() >> 12), (int)(rng() % 400) - 200), at(c, e));
        quotient(at(one | (rng() >> 12), 1), at(top, e));
    }
    for (double z : {0.0, -0.0})
        for (double c : {1.0, 0.7225, 0x1.fffffffffffffp-1, 0x1p-300, 0x1p900}) quotient(z, c);
    const double edge[] = {0.0, 0x1p-1074, 0x1.8p-1060, 0x1p-1042, 0x1.23456789abcdep-1030, 0x1p-1022, 0x1p-1021,
                           0x1.fffffffffffffp-961, 0x1p-960, 0x1.3p-900, 0x1p-600, 0x1.fffffffffffffp-1, 1.0, 1.7,
                           0x1p59, 0x1.8p60, 0x1p450, 0x1p900, 0x1.fffffffffffffp1020, 0x1p1022, 0x1.4p1023,
                           std::numeric_limits<double>::infinity(), std::numeric_limits<double>::quiet_NaN()};
    std::uniform_real_distribution<double> w(1.0, 2.0);
    for (double x : edge)
        for (double c : edge)
            for (int i = 0; i < 60; ++i) {
                const double f = i ? w(rng) : 1.0, g = i ? w(rng) : 1.0;
                guarded(x * f, c * g);
                guarded(-x * f, c * g);
            }
    // the one kind of divisor that recip_rn may miss is no square: none of the
    // doubles around 2^(1/2) and below 2 (and so of no other binade) gives it
    bool missed = false;
    for (int i = 0; i < 100; ++i) missed = missed || recip_rn(0x1.fffffffffffffp0) != 1.0;
    check(missed, "all bits set", 1.0, 0x1.fffffffffffffp0);
    for (double s : {std::sqrt(2.0), 2.0, 1.0})
        for (int k = -64; k <= 64; ++k) {
            const double r = s + k * 0x1p-52, c = r * r;
            uint64_t b;
            std::memcpy(&b, &c, 8);
            check((b & top >> 1) != top >> 1, "square", r, 1.0);
        }
    std::printf("%ld checked, %ld wrong\n", checked, wrong);
    return wrong != 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a host compiler")
def test_quotients_are_the_ieee_ones(tmp_path):
    (tmp_path / "q.cpp").write_text(PROGRAM)
    exe = tmp_path / "q"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(CSRC), str(tmp_path / "q.cpp"), "-o",
                    str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
