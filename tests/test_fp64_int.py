"""The integer-pipe double-precision operations (fp64_int.cuh) against the host's IEEE operations.

The header's code is the same on the device and the host; the device's reciprocal and root estimates are
off by two units in the last place at most, and a test moves the host's stand-ins by as much."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

DRIVER = r"""
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
#include "fp64_int.cuh"
using fi::bits;
static bool same(double a, double b) { return bits(a) == bits(b) || (a != a && b != b); }
int main(int, char** v) {
    std::mt19937_64 g(std::atoi(v[1]));
    const double sp[] = {0., -0., INFINITY, -INFINITY, NAN, -NAN, 5e-324, -5e-324, 0x1p-1022, 0x1.fffffffffffffp+1023,
                         1, -1, 1e-200, -1e-200, 1e200};
    const uint64_t frac = 0xfffffffffffffull;
    for (long i = 0; i < 3000000; i++) {
        uint64_t a = g(), b = g();
        const int mode = i % 9;  // any bits; then moderate exponents with random, short, near-2, near-1 and
                                 // equal-but-for-units significands, zeros, special values
        if (mode >= 2) {
            a = (a & 0x800fffffffffffffull) | ((1023 - 60 + g() % 120) << 52);
            b = (b & 0x800fffffffffffffull) | ((1023 - 60 + g() % 120) << 52);
        }
        if (mode == 3) { b &= ~((1ull << g() % 53) - 1); a &= ~((1ull << g() % 53) - 1); }
        if (mode == 4) { b |= frac & ~(g() % 8); if (g() & 1) a |= frac & ~(g() % 8); }
        if (mode == 5) { b = (b & ~frac) | g() % 16; if (g() & 1) a = (a & ~frac) | g() % 16; }
        if (mode == 6) a = (((b & frac) + g() % 5 - 2) & frac) | (1023ull << 52);
        if (mode == 7 && (i & 8)) a &= 1ull << 63;
        double x = fi::from_bits(a), y = fi::from_bits(b);
        if (mode == 2) a = (a & 0x800fffffffffffffull) | ((1023 - 152 + g() % 285) << 52);  // FP32's range and edges
        if (mode == 2 && (i & 16)) a = (a & ~0x3fffffffull) | 0x10000000ull;  // ties of the conversion
        if (mode == 2) x = fi::from_bits(a);
        if (mode == 8) { x = sp[g() % 15]; if (g() & 1) y = sp[g() % 15]; if (g() % 7 == 0) x = y; }
        const double mm = (x * y <= 0) ? 0.0 : (std::fabs(x) < std::fabs(y) ? x : y);
        const double m = fi::minmod(x, y);
        const bool cmp = fi::lt(x, y) == (x < y) && fi::le(x, y) == (x <= y) && fi::lt0(x) == (x < 0) &&
                         fi::gt0(x) == (x > 0) && fi::ge0(x) == (x >= 0) && fi::le0(x) == (x <= 0) &&
                         fi::abs_lt(x, y) == (std::fabs(x) < std::fabs(y));
        if (!same(fi::div(x, y), x / y) || !cmp || !(same(m, mm) || (m == 0 && mm == 0)) ||
            !same(fi::half(x), 0.5 * x) || !same(fi::to_float(x), (float)x) ||
            !same(fi::to_double((float)y), (double)(float)y)) {
            std::printf("%a %a\n", x, y);
            return 1;
        }
        if (mode == 6) x = fi::from_bits(bits(x * x) + g() % 5 - 2);  // squares and their neighbours
        if (!same(fi::sqrt(x), std::sqrt(x))) {
            std::printf("sqrt %a\n", x);
            return 1;
        }
    }
    return 0;
}
"""


@pytest.mark.parametrize("ulp", [-2, 0, 2])
def test_integer_operations_are_ieee(tmp_path, ulp):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(DRIVER)
    subprocess.run(["g++", "-std=c++17", "-O2", f"-DFI_ESTIMATE_ULP={ulp}",
                    "-I", os.path.join(ROOT, "deorbit_gb300", "csrc"), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe), str(ulp + 3)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
