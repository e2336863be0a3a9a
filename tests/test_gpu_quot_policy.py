"""The friction update's quotient as each policy forms it (quot, csrc/stencil.cuh)
against the IEEE division, bit for bit (tolerance 0): dividends of every class
the wavefield holds (zeros of both signs, subnormal, ordinary, infinite, NaN)
over ordinary divisors, in 2D and 3D.  And quot_y in FP64 where its results are
subnormal or nearly so: dividends of every size down to the smallest, by
spacings (doubles widened from floats) and by full significands, a part of them
next to a midpoint of two subnormal neighbours."""
import subprocess
from pathlib import Path

import pytest

from mixedprecisionfaracoustic_b200 import build as B

pytestmark = pytest.mark.gpu
CSRC = Path(B.CSRC)

PROGRAM = r"""
#include "stencil.cuh"
#include <cstdio>
using namespace bpk;
__device__ unsigned rnd(unsigned long long& s) { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return (unsigned)(s >> 16); }
__device__ bool same(float a, float b) { return (a != a && b != b) || __float_as_int(a) == __float_as_int(b); }
__global__ void k(unsigned long long* bad) {
    unsigned long long s = (blockIdx.x * 256ull + threadIdx.x + 1) * 0x9E3779B97F4A7C15ull;
    for (int i = 0; i < 8; i++) rnd(s);
    for (int i = 0; i < 256; i++) {
        unsigned a = rnd(s);
        const unsigned b = (rnd(s) & 0x807fffffu) | ((97u + rnd(s) % 60u) << 23);
        const int c = i & 7;
        if (c == 0) a &= 0x80000000u;                         // zero
        else if (c == 1) a &= 0x807fffffu;                    // subnormal
        else if (c == 2) a = (a & 0x807fffffu) | ((1u + rnd(s) % 40u) << 23);
        else if (c == 3) a = (a & 0x80000000u) | 0x7f800000u;
        const float x = __uint_as_float(a), y = __uint_as_float(b), e = __fdiv_rn(x, y);
        if (!same(quot<PolF32, 2>(x, y), e)) atomicAdd(bad, 1ull);
        if (!same(quot<PolF32, 3>(x, y), e)) atomicAdd(bad + 1, 1ull);
        if (!same(quot<PolB24, 2>(x, y), e)) atomicAdd(bad + 2, 1ull);
        if (!same(quot<PolB24, 3>(x, y), e)) atomicAdd(bad + 3, 1ull);
    }
}
int main() {
    unsigned long long* b;
    cudaMallocManaged(&b, 32);
    b[0] = b[1] = b[2] = b[3] = 0;
    k<<<2048, 256>>>(b);
    if (cudaDeviceSynchronize() != cudaSuccess) return 2;
    printf("%llu %llu %llu %llu\n", b[0], b[1], b[2], b[3]);
}
"""


def test_friction_quotient_of_each_policy(tmp_path):
    (tmp_path / "q.cu").write_text(PROGRAM)
    exe = tmp_path / "q"
    subprocess.run([B._nvcc(), *B._host_cxx(), "-std=c++17", "-O3", *B.ARCH, "-diag-suppress", "177", "-I", str(CSRC),
                    "-o", str(exe), str(tmp_path / "q.cu")], check=True, capture_output=True, timeout=600)
    r = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=300)
    assert r.stdout.split() == ["0"] * 4


SMALL = r"""
#include "stencil.cuh"
#include <cstdio>
using namespace bpk;
__device__ unsigned long long rnd(unsigned long long& s) { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; }
__global__ void k(unsigned long long* n) {
    unsigned long long s = (blockIdx.x * 256ull + threadIdx.x + 1) * 0x9E3779B97F4A7C15ull;
    for (int i = 0; i < 8; i++) rnd(s);
    for (int i = 0; i < 512; i++) {
        const unsigned long long u = rnd(s);
        double b = i & 1 ? (double)__uint_as_float((unsigned)(u & 0x7fffff) | ((107u + (unsigned)(u >> 32) % 41u) << 23))
                         : ldexp(1.0 + (double)(u >> 12) * 0x1p-52, (int)(u % 41) - 20);
        const unsigned long long v = rnd(s);
        double a = ldexp(1.0 + (double)(v >> 12) * 0x1p-52, -1080 + (int)(v % 120));
        if ((i & 6) == 2) a = ldexp((double)(2 * (v % 4096) + 1), -1075) * b;      // about a midpoint of results
        if ((i & 6) == 4) a = __longlong_as_double((long long)(v % 4096));         // the smallest dividends
        if (v >> 63) a = -a;
        const double e = __ddiv_rn(a, b), q = quot_y<double>(a, b, __drcp_rn(b));
        if (__double_as_longlong(e) != __double_as_longlong(q)) atomicAdd(n, 1ull);
        if (e != 0.0 && fabs(e) < 0x1p-1022) atomicAdd(n + 1, 1ull);
    }
}
int main() {
    unsigned long long* n;
    cudaMallocManaged(&n, 16);
    n[0] = n[1] = 0;
    k<<<2048, 256>>>(n);
    if (cudaDeviceSynchronize() != cudaSuccess) return 2;
    printf("%llu %llu\n", n[0], n[1]);
}
"""


def test_fp64_quotients_with_subnormal_results(tmp_path):
    (tmp_path / "q.cu").write_text(SMALL)
    exe = tmp_path / "q"
    subprocess.run([B._nvcc(), *B._host_cxx(), "-std=c++17", "-O3", *B.ARCH, "-diag-suppress", "177", "-I", str(CSRC),
                    "-o", str(exe), str(tmp_path / "q.cu")], check=True, capture_output=True, timeout=600)
    r = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=300)
    wrong, subnormal = map(int, r.stdout.split())
    assert wrong == 0 and subnormal > 1 << 25
