"""quot_y / recip (csrc/stencil.cuh): the phase kernels' quotients without the
divide routine must equal the IEEE ones bit for bit (tolerance 0).  A small
program built around the header compares them on 2^28 operand pairs per class:
any dividend (subnormal, infinite, NaN) against ordinary divisors, both near 1,
tiny dividends (subnormal quotients, where a second rounding would show), and
divisors just below a power of two; in FP64 also dividends near the smallest."""
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
__device__ unsigned long long rnd(unsigned long long& s) { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; }
template <class R> __device__ bool same(R a, R b) { return (a != a && b != b) || (a == b && signbit(a) == signbit(b)); }
__global__ void k(int mode, unsigned long long* bad) {
    unsigned long long s = (blockIdx.x * 256ull + threadIdx.x + 1) * 0x9E3779B97F4A7C15ull;
    for (int i = 0; i < 8; i++) rnd(s);
    for (int i = 0; i < 1024; i++) {
        unsigned a = (unsigned)rnd(s), b = (unsigned)rnd(s);
        if (mode == 0) b = (b & 0x007fffff) | ((97 + (b >> 23) % 60) << 23);
        else if (mode == 1) { a = (a & 0x807fffff) | ((117 + ((a >> 23) & 15)) << 23); b = (b & 0x007fffff) | ((117 + ((b >> 23) & 15)) << 23); }
        else if (mode == 2) { a &= 0x80ffffff; b = (b & 0x007fffff) | ((120 + ((b >> 23) & 31)) << 23); }
        else { a = (a & 0x807fffff) | (127 << 23); b = (0x7fffff - (b & 15)) | (127 << 23); }
        const float fa = __uint_as_float(a), fb = __uint_as_float(b), e = __fdiv_rn(fa, fb);
        if (!same(quot_y<float>(fa, fb, recip(fb)), e)) atomicAdd(bad, 1ull);
        if (!same(quot_y<float>(fa, fb, __fdiv_rn(1.0f, fb)), e)) atomicAdd(bad, 1ull);
        double da = (double)fa * (1.0 + 1e-9 * (double)(rnd(s) >> 40)), db = (double)fb * (1.0 + 1e-9 * (double)(rnd(s) >> 40));
        if (mode == 0) da = __longlong_as_double(rnd(s));
        if (mode == 2) da *= 1e-270;
        if (!same(quot_y<double>(da, db, 1.0 / db), da / db)) atomicAdd(bad + 1, 1ull);
    }
}
int main() {
    unsigned long long* b;
    cudaMallocManaged(&b, 16);
    for (int m = 0; m < 4; m++) {
        b[0] = b[1] = 0;
        k<<<1024, 256>>>(m, b);
        if (cudaDeviceSynchronize() != cudaSuccess) return 2;
        printf("%d %llu %llu\n", m, b[0], b[1]);
    }
}
"""


def test_quotients_equal_the_division(tmp_path):
    (tmp_path / "q.cu").write_text(PROGRAM)
    exe = tmp_path / "q"
    subprocess.run([B._nvcc(), *B._host_cxx(), "-std=c++17", "-O3", *B.ARCH, "-diag-suppress", "177", "-I", str(CSRC),
                    "-o", str(exe), str(tmp_path / "q.cu")], check=True, capture_output=True, timeout=600)
    r = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=300)
    rows = [tuple(map(int, line.split())) for line in r.stdout.splitlines()]
    assert rows == [(m, 0, 0) for m in range(4)]


@pytest.mark.parametrize("dx", [5.0, 5.02465773, 4.0])
@pytest.mark.parametrize("order", [2, 4])
def test_reference_rounding_at_spacings_of_each_kind(dx, order):
    """A spacing the two-operation division holds for, one it does not (every
    difference through quot_y), and a power of two: against the oracle's
    reference arithmetic, <= 1e-5 as everywhere (test_gpu_parity.py)."""
    import numpy as np
    from mixedprecisionfaracoustic_b200 import Simulation
    from oracle import oracle as O
    from test_gpu_parity import small_2d
    cfg, med = small_2d(order, "fp32", nx=90, nz=61, nt=200)
    cfg.dx, cfg.rounding = dx, "reference"
    with Simulation(cfg, med) as s:
        s.run(cfg.nt)
        got = {c: s.traces(c) for c in ("txx", "vux", "p")}
    o = O.Oracle(cfg, med, O.REF32)
    o.run(cfg.nt)
    for c, g in got.items():
        want = np.asarray(o.traces(c), np.float64)
        assert np.linalg.norm(g - want) <= 1e-5 * np.linalg.norm(want), c
