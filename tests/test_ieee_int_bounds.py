"""The integer-pipe division and roots (csrc/ieee_int.h) on the host with the
FP32 estimates moved over the whole of the device's error: a reciprocal by up to
one unit in the last place, a reciprocal square root by up to two (its bound,
2^-22.9 relative, is 2.1 units of a value next to 1)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "ieee_int.h"
#include <cstdio>
#include <cstdlib>
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
int main(int, char **argv) {
    std::mt19937_64 g(7);
    const int rcp = atoi(argv[1]), rsqrt = atoi(argv[2]);
    long bad = 0;
    for (long i = 0; i < 3000000; ++i) {
        double a = ii_double(((900 + g() % 250) << 52) | frac(g));
        double b = ii_double(((900 + g() % 250) << 52) | frac(g));
        if (i % 16 == 1) a = b * ii_double(0x3ff0000000000000ULL | frac(g)); /* quotients next to a double */
        const double s = ii_double(0x3ff0000000000000ULL | frac(g));
        double q = ii_double(((1022 + g() % 4) << 52) | frac(g));
        if (i % 16 == 3) q = s * s; /* roots next to a double */
        ii_nudge() = rcp;
        bad += ii_bits(ii_div(a, b)) != ii_bits(a / b);
        ii_nudge() = rsqrt;
        bad += ii_bits(ii_sqrt(q)) != ii_bits(sqrt(q));
        bad += ii_bits(ii_inv_sqrt(q)) != ii_bits(1.0 / sqrt(q));
    }
    printf("%ld\n", bad);
    return bad != 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("ieee")
    (d / "t.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "network_relaxation_gb300", "csrc"), str(d / "t.cpp"), "-o", str(d / "t")], check=True)
    return str(d / "t")


@pytest.mark.parametrize("rcp,rsqrt", [(-1, -2), (1, 2), (0, -1), (0, 1), (0, 0)])
def test_estimates_moved(program, rcp, rsqrt):
    out = subprocess.run([program, str(rcp), str(rsqrt)], stdout=subprocess.PIPE, text=True)
    assert out.returncode == 0, out.stdout
