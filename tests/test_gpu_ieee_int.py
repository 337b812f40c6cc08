"""The integer-pipe division and roots (csrc/ieee_int.h) on the device: the FP32
estimates over every significand there is, and the results against the device's
IEEE operations, bit for bit, over random and extreme significands."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "ieee_int.h"
#include <cstdio>
using namespace nr;

/* largest distance of an estimate from the correctly rounded FP32 value, in
 * units of 2^-24 (its last place in [1/2, 1)), over all FP32 arguments */
__global__ void estimates(unsigned *far) {
    const unsigned n = 1u << 24;
    unsigned rcp = 0, rsq = 0;
    for (unsigned k = blockIdx.x * blockDim.x + threadIdx.x; k <= n; k += gridDim.x * blockDim.x) {
        const unsigned f = 0x3f800000u + k; /* 1 .. 4 */
        const double x = (double)__uint_as_float(f);
        auto dist = [](unsigned q, double exact) {
            const double r = rint(exact * 16777216.0); /* to 24 bits */
            const double d = fabs((double)(q >> 8) - fmin(fmax(r, 8388608.0), 16777215.0));
            return (unsigned)d;
        };
        if (k <= 1u << 23) rcp = max(rcp, dist(ii_rcp_q32(f), 1.0 / x));
        rsq = max(rsq, dist(ii_rsqrt_q32(f), 1.0 / sqrt(x)));
    }
    atomicMax(far, rcp);
    atomicMax(far + 1, rsq);
}

__device__ unsigned long long mix(unsigned long long z) { /* SplitMix64's finaliser */
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    return z ^ (z >> 31);
}
struct Rng {
    unsigned long long s;
    __device__ unsigned long long operator()() { return mix(s += 0x9E3779B97F4A7C15ULL); }
};
__device__ unsigned long long frac(Rng &g) {
    const unsigned long long m = g() & kIiFrac, r = g();
    switch (r % 10) { /* ends of the range, few bits, long runs of ones */
    case 0: return 0;
    case 1: return kIiFrac - (r >> 32) % 64;
    case 2: return (r >> 32) % 64;
    case 3: return m & ~0ULL << ((r >> 32) % 52);
    case 4: return (m | ((1ULL << ((r >> 32) % 52)) - 1)) & kIiFrac;
    }
    return m;
}
__device__ bool same(double a, double b) { return ii_bits(a) == ii_bits(b) || (a != a && b != b); }
__global__ void results(unsigned long long *bad, long n) {
    unsigned long long wrong[3] = {0, 0, 0};
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        Rng g{mix(i + 1)};
        double a = ii_double((900 + g() % 250) << 52 | frac(g) | (g() & 1) << 63);
        double b = ii_double((900 + g() % 250) << 52 | frac(g) | (g() & 1) << 63);
        if (i % 16 == 0) a = ii_double(g()), b = ii_double(g()); /* any bits */
        if (i % 16 == 1) a = b * ii_double(0x3ff0000000000000ULL | frac(g)); /* quotients next to a double */
        double q = fabs(a);
        const double s = ii_double(0x3ff0000000000000ULL | frac(g));
        if (i % 16 == 3) q = s * s; /* roots next to a double */
        if (i % 16 == 4) q = ii_double(((1022 + g() % 4) << 52) | frac(g)); /* [1/2, 8) */
        wrong[0] += !same(ii_div(a, b), a / b);
        wrong[1] += !same(ii_sqrt(q), sqrt(q));
        wrong[2] += !same(ii_inv_sqrt(q), 1.0 / sqrt(q));
    }
    for (int k = 0; k < 3; ++k)
        if (wrong[k]) atomicAdd(bad + k, wrong[k]);
}

int main() {
    unsigned long long *buf, h[4];
    if (cudaMalloc(&buf, sizeof h) != cudaSuccess || cudaMemset(buf, 0, sizeof h) != cudaSuccess) return 2;
    estimates<<<1024, 256>>>((unsigned *)buf);
    results<<<1024, 256>>>(buf + 1, 1L << 27);
    if (cudaMemcpy(h, buf, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
    printf("%u %u %llu %llu %llu\n", (unsigned)h[0], (unsigned)(h[0] >> 32), h[1], h[2], h[3]);
    return 0;
}
"""


def test_estimates_and_results(cuda, tmp_path):
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    src = tmp_path / "t.cu"
    src.write_text(PROGRAM)
    subprocess.run([nvcc if os.path.exists(nvcc) else shutil.which("nvcc"), "-gencode", "arch=compute_103a,code=sm_103a",
                    "-O3", "-std=c++17", "--fmad=false", "-I", os.path.join(ROOT, "network_relaxation_gb300", "csrc"),
                    str(src), "-o", str(tmp_path / "t")], check=True)
    out = subprocess.run([str(tmp_path / "t")], stdout=subprocess.PIPE, text=True, check=True).stdout
    rcp, rsqrt, div, root, inv = (int(v) for v in out.split())
    assert (div, root, inv) == (0, 0, 0), out
    # what the host test sweeps (test_ieee_int_bounds.py)
    assert rcp <= 1 and rsqrt <= 2, out
    print(out)
