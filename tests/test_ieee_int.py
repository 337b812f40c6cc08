"""The integer-pipe division and roots (csrc/ieee_int.h), compiled for the
host, against the host's IEEE operations: the same bits."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "ieee_int.h"
#include <cstdio>
#include <random>
using namespace nr;
static uint64_t frac(std::mt19937_64 &g) {
    uint64_t m = g() & kIiFrac;
    switch (g() % 10) { /* ends of the range, few bits, long runs of ones */
    case 0: return 0;
    case 1: return kIiFrac - g() % 64;
    case 2: return g() % 64;
    case 3: return m & ~0ULL << (g() % 52);
    case 4: return (m | ((1ULL << (g() % 52)) - 1)) & kIiFrac;
    }
    return m;
}
static bool same(double a, double b) { return ii_bits(a) == ii_bits(b) || (a != a && b != b); }
int main() {
    std::mt19937_64 g(5);
    long bad = 0;
    for (long i = 0; i < 4000000; ++i) {
        ii_nudge() = (int)(g() % 3) - 1; /* the FP32 estimate off by up to 1.5 ulp */
        double a = ii_double(((900 + g() % 250) << 52) | frac(g) | (g() & 1) << 63);
        double b = ii_double(((900 + g() % 250) << 52) | frac(g) | (g() & 1) << 63);
        if (i % 16 == 0) a = ii_double(g()), b = ii_double(g()); /* any bits: zeros, subnormals, inf, NaN */
        if (i % 16 == 1) a = b * ii_double(0x3ff0000000000000ULL | frac(g)); /* quotients next to a double */
        if (i % 64 == 2) a = i & 64 ? 0.0 : -0.0;
        double q = fabs(a), s = ii_double(0x3ff0000000000000ULL | frac(g));
        if (i % 16 == 3) q = s * s; /* roots next to a double */
        bad += !same(ii_div(a, b), a / b) + !same(ii_sqrt(q), sqrt(q)) + !same(ii_inv_sqrt(q), 1.0 / sqrt(q));
        bad += !same(ii_sqrt(a), sqrt(a)) + !same(ii_inv_sqrt(a), 1.0 / sqrt(a));
        bad += a == a && (ii_negative(a) != (a < 0.0) || ii_is_zero(a) != (a == 0.0)); /* a NaN may answer either way */
    }
    printf("%ld\n", bad);
    return bad != 0;
}
"""


def test_integer_division_and_roots_are_ieee(tmp_path):
    src = tmp_path / "t.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "t"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "network_relaxation_gb300", "csrc"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], stdout=subprocess.PIPE, text=True)
    assert out.returncode == 0, out.stdout
