"""div_by (sphere_b200/csrc/tagged.cuh) against the division it stands for.

The Darcy kernels divide by the cell widths through their reciprocals; their
results equal the division's bit for bit.  A small program compares the two over
operands whose bits are drawn, and over the edges: zeros, infinities, NaN, the
smallest and largest magnitudes, quotients that are exact, divisors that are
powers of two or have all mantissa bits set.
"""
import os
import subprocess

import pytest

from sphere_b200 import build

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include "tagged.cuh"

__host__ __device__ inline unsigned long long mix(unsigned long long z)
{
    z += 0x9e3779b97f4a7c15ull;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}

__host__ __device__ inline double value(unsigned long long bits)
{
    double v;
    memcpy(&v, &bits, 8);
    return v;
}

// whether case i differs: the divisor is a length between 2^-40 and 2^40
__host__ __device__ inline bool differs(unsigned long long i)
{
    const unsigned long long a = mix(2 * i), b = mix(2 * i + 1), mant = (1ull << 52) - 1;
    unsigned long long dm = b & mant;
    if (i % 7 == 1) dm = 0;                          // a power of two
    if (i % 7 == 2) dm = mant - (b >> 60);           // all bits set, or nearly
    if (i % 7 == 3) dm = b >> 60;                    // just above a power of two
    const double d = value((1023ull - 40 + (b >> 52) % 81) << 52 | dm);
    double x = value(a);                             // any bits: subnormal, infinite, NaN
    if (i % 5 == 1) x = d * (double)(long long)(a % 2000001 - 1000000);
    if (i % 5 == 2) x = value((a & (mant | 1ull << 63)) | (1023ull - 60 + (a >> 52) % 121) << 52);
    if (i % 5 == 3) x = value(((a >> 60) << 62) | (a & mant & ~0xffull));
    if (i % 1001 == 0) x = i % 2 ? 0.0 : -0.0;
    const double q = x / d, r = sphb::div_by(x, d, 1.0 / d);
    unsigned long long p, s;
    memcpy(&p, &q, 8);
    memcpy(&s, &r, 8);
    return p != s && !(q != q && r != r);
}

__global__ void count(unsigned long long n, unsigned long long *bad)
{
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n;
         i += (unsigned long long)gridDim.x * blockDim.x)
        if (differs(i)) atomicAdd(bad, 1ull);
}

int main(int argc, char **argv)
{
    const unsigned long long n = strtoull(argv[1], nullptr, 10);
    unsigned long long bad = 0;
    if (argc > 2) {
        unsigned long long *d = nullptr;
        if (cudaMalloc(&d, 8) != cudaSuccess || cudaMemset(d, 0, 8) != cudaSuccess) return 2;
        count<<<1184, 256>>>(n, d);
        if (cudaMemcpy(&bad, d, 8, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
        cudaFree(d);
    } else {
        for (unsigned long long i = 0; i < n; ++i) bad += differs(i);
    }
    std::printf("%llu\n", bad);
    return 0;
}
"""


def mismatches(tmp_path, n, *mode):
    src, exe = tmp_path / "div_by.cu", tmp_path / "div_by"
    src.write_text(PROGRAM)
    subprocess.check_call([build.nvcc(), "-O2", "-std=c++17", "-fmad=false", "-Xcompiler", "-ffp-contract=off",
                           *build.ARCH, "-I", build.CSRC, str(src), "-o", str(exe)])
    out = subprocess.run([str(exe), str(n), *mode], stdout=subprocess.PIPE, check=True, env=os.environ)
    return int(out.stdout)


def test_div_by_equals_the_division(tmp_path):
    assert mismatches(tmp_path, 20_000_000) == 0


@pytest.mark.gpu
def test_div_by_equals_the_division_on_the_device(tmp_path):
    assert mismatches(tmp_path, 2_000_000_000, "device") == 0
