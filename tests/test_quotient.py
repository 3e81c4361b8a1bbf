"""Quotients from a shared reciprocal against the division, bit for bit: random
operands, ones a few units in the last place from a multiple of the divisor or
from halfway between two quotients, divisors just above and below powers of two,
the ends of the range that takes the reciprocal, and what it must leave to the
division (zero, infinite, tiny and huge divisors, numbers that are none)."""
from host_program import run

PROGRAM = r"""
#include "quotient.cuh"
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>
static unsigned long long bits(double v) { unsigned long long b; std::memcpy(&b, &v, 8); return b; }
static double from(unsigned long long b) { double v; std::memcpy(&v, &b, 8); return v; }
// the same number (of zeros the sign does not count, of NaNs nothing)
static bool same(double a, double b) { return (a != a && b != b) || (a == 0.0 && b == 0.0) || bits(a) == bits(b); }
static long wrong = 0, tried = 0, direct = 0;
static void check(double a, double b) {
    volatile double d = b, n = a;
    const double want = n / d, got = mcm::divide(a, b, 1.0 / d);
    ++tried;
    if (mcm::dividend_in_range(a) && mcm::divisor_in_range(b)) ++direct;
    if (!same(want, got) && wrong++ < 5) std::fprintf(stderr, "%a / %a: %a, not %a\n", a, b, got, want);
}
int main() {
    std::mt19937_64 rng(7);
    auto number = [&](int lo, int hi) {
        const unsigned long long e = 1023 + lo + (long long)(rng() % (unsigned)(hi - lo + 1));
        return from((rng() >> 63 << 63) | e << 52 | rng() >> 12);
    };
    for (long k = 0; k < 1000000; ++k) {
        check(number(-60, 60), number(-60, 60));
        check(number(-499, 499), number(-499, 499));
        // near a multiple, and near the middle between two neighbouring quotients
        const double b = number(-300, 300), q = number(-150, 150);
        check(from(bits(q * b) + rng() % 7 - 3), b);
        const double half = std::fma(q, b, b * (from(bits(q) + 1) - q) * 0.5);
        check(from(bits(half) + rng() % 5 - 2), b);
        // divisors whose fraction is nearly all zeros or all ones
        const double edge = from((bits(number(-300, 300)) & 0xfff0000000000000ull) + rng() % 9 - 4);
        check(number(-300, 300), edge);
        check(from(bits(edge * q) + rng() % 5 - 2), edge);
    }
    const double inf = std::numeric_limits<double>::infinity(), nan = std::numeric_limits<double>::quiet_NaN();
    const double ends[] = {0.0, 5e-324, 2.2e-308, 0x1p-501, 0x1p-500, 0x1.8p-499, 1e-30, 1.0, 1e30, 0x1p499, 0x1p500, 0x1p501,
                           1.7e308, inf, nan};
    for (double a : ends)
        for (double b : ends)
            for (int s = 0; s < 4; ++s) check(s & 1 ? -a : a, s & 2 ? -b : b);
    std::printf("%ld %ld %ld\n", wrong, tried, direct);
}
"""


def test_quotients_are_the_divisions(tmp_path):
    wrong, tried, direct = (int(v) for v in run(str(tmp_path), PROGRAM).split())
    assert wrong == 0 and tried > 6000000 and direct > 0.9 * tried
