"""Division by a common divisor (sph_gb300/csrc/sph_divide.h) against the division itself, bit for bit, on the CPU: the
header is plain C++ whose operations round alike on both.  Random operands of all magnitudes, significands whose
quotients lie next to the middle of two results, and operands at and beyond the ends of the range."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "sph_divide.h"
#include <cstdio>
#include <random>
#include <limits>
static long bad = 0, done = 0;
static void check(double x, double b)
{
    volatile double vb = b, vx = x;
    const double want = vx / vb;
    double got;
    ++done;
    if (!sph::quotient(x, sph::divisor(b), &got)) {
        // (left to the caller: no operands of ordinary size among these)
        const double ax = std::fabs(x), ab = std::fabs(b);
        if ((ax >= 0x1p-799 && ax < 0x1p799 || x == 0) && ab >= 0x1p-99 && ab < 0x1p99) ++bad;
        return;
    }
    if (x == 0 && got == 0) return;  // of either sign
    if (std::memcmp(&want, &got, 8) != 0 && !(want != want && got != got)) {
        if (++bad <= 10) std::printf("%a / %a = %a, not %a\n", x, b, want, got);
    }
}
int main()
{
    std::mt19937_64 rng(7);
    std::uniform_real_distribution<double> sig(1.0, 2.0);
    auto any = [&](int lo, int hi) { return std::ldexp(sig(rng) * (rng() & 1 ? -1.0 : 1.0), lo + (int)(rng() % (hi - lo + 1))); };
    for (int k = 0; k < 3000000; ++k) check(any(-60, 20), std::fabs(any(-25, 3)));
    for (int k = 0; k < 1000000; ++k) check(any(-1074, 1023), any(-1074, 1023));
    for (int k = 0; k < 1000000; ++k) check(any(-860, -740), any(-110, 110)), check(any(740, 860), any(-110, 110));
    // quotients close to halfway between two doubles: x = b (q + ulp / 2) rounded, and its neighbours
    for (int k = 0; k < 1000000; ++k) {
        const double b = sig(rng), q = sig(rng);
        double x = (double)((long double)b * ((long double)q + 0x1p-53L));
        for (int n = 0; n < 3; ++n) {
            check(x, b);
            x = std::nextafter(x, n == 0 ? 0.0 : 10.0);
        }
    }
    // significands of many ones and few ones
    for (int k = 0; k < 53; ++k)
        for (int j = 0; j < 53; ++j)
            for (int s = -1; s <= 1; s += 2)
                check(1.0 + s * std::ldexp(1.0, -k - 1), 1.0 + s * std::ldexp(1.0, -j - 1)), check(2.0 - std::ldexp(1.0, -k), 1.0 + std::ldexp(1.0, -j));
    const double inf = std::numeric_limits<double>::infinity(), nan = std::nan("");
    const double edge[] = {0.0, -0.0, 5e-324, -5e-324, 2.2250738585072014e-308, 0x1p-801, 0x1p-800, 0x1p800, 0x1p801, 0x1p-101, 0x1p-100, 0x1p100, 0x1p101, 1.0, 3.0, -7.0,
                           1.7976931348623157e308, inf, -inf, nan};
    for (double x : edge)
        for (double b : edge) check(x, b);
    std::printf("%ld of %ld differ\n", bad, done);
    return bad != 0;
}
"""


def test_quotients_are_the_divisions(tmp_path):
    src, exe = tmp_path / "divide.cpp", str(tmp_path / "divide")
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", os.path.join(ROOT, "sph_gb300", "csrc"), "-o", exe, str(src)],
                   check=True, capture_output=True, text=True)
    p = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stdout
