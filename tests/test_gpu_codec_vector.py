"""decode_ch4 / encode_ch4 (csrc/common.cuh), the four-value COMP16 codec of the
phase kernels, against the scalar decode_ch / encode_ch that test_gpu_codec.py
holds to the oracle: every (hi, lo) pair and every float, bit for bit."""
import subprocess

import pytest

from mixedprecisionfaracoustic_b200 import build as B

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include "common.cuh"
#include <cstdio>
using namespace bpk;
__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b) || (a != a && b != b); }
__global__ void dec(unsigned long long* bad) {          // 2^22 threads x 4 pairs
    const unsigned t = blockIdx.x * 256 + threadIdx.x;
    unsigned short h[4]; signed char l[4];
    for (int j = 0; j < 4; j++) { const unsigned p = (t * 4 + j) * 2654435761u >> 8; h[j] = p & 0xffff; l[j] = (signed char)(p >> 16); }
    float v[4];
    decode_ch4(make_uint2(h[0] | h[1] << 16, h[2] | (unsigned)h[3] << 16),
               (unsigned char)l[0] | (unsigned char)l[1] << 8 | (unsigned char)l[2] << 16 | (unsigned)(unsigned char)l[3] << 24, v);
    for (int j = 0; j < 4; j++)
        if (!same(v[j], decode_ch(__ushort_as_half(h[j]), l[j]))) atomicAdd(bad, 1ull);
    for (int j = 0; j < 4; j++) {                       // and each hi with each lo, in order
        const unsigned p = t * 4 + j;
        h[j] = p >> 8; l[j] = (signed char)(p & 255);
    }
    decode_ch4(make_uint2(h[0] | h[1] << 16, h[2] | (unsigned)h[3] << 16),
               (unsigned char)l[0] | (unsigned char)l[1] << 8 | (unsigned char)l[2] << 16 | (unsigned)(unsigned char)l[3] << 24, v);
    for (int j = 0; j < 4; j++)
        if (!same(v[j], decode_ch(__ushort_as_half(h[j]), l[j]))) atomicAdd(bad, 1ull);
}
__global__ void enc(unsigned long long* bad) {          // 2^30 chunks of 4 floats
    const unsigned step = gridDim.x * 256;
    for (unsigned t = blockIdx.x * 256 + threadIdx.x; t < 1u << 30; t += step) {
        float v[4];
        for (int j = 0; j < 4; j++) v[j] = __uint_as_float((unsigned)j << 30 | (t * 2654435761u & 0x3fffffffu));
        uint2 h; unsigned l;
        encode_ch4(v, h, l);
        for (int j = 0; j < 4; j++) {
            __half hj; int8_t lj;
            encode_ch(v[j], hj, lj);
            const unsigned g = (j < 2 ? h.x : h.y) >> 16 * (j & 1) & 0xffff;
            if (g != __half_as_ushort(hj) || (l >> 8 * j & 255) != (unsigned char)lj) atomicAdd(bad + 1, 1ull);
        }
    }
}
int main() {
    unsigned long long* b;
    cudaMallocManaged(&b, 16);
    b[0] = b[1] = 0;
    dec<<<1 << 14, 256>>>(b);
    enc<<<148 * 8, 256>>>(b);
    if (cudaDeviceSynchronize() != cudaSuccess) return 2;
    printf("%llu %llu\n", b[0], b[1]);
}
"""


def test_vector_codec_equals_the_scalar_one(tmp_path):
    (tmp_path / "c.cu").write_text(PROGRAM)
    exe = tmp_path / "c"
    subprocess.run([B._nvcc(), *B._host_cxx(), "-std=c++17", "-O3", *B.ARCH, "-diag-suppress", "177", "-I", str(B.CSRC),
                    "-o", str(exe), str(tmp_path / "c.cu")], check=True, capture_output=True, timeout=600)
    r = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=300)
    assert r.stdout.split() == ["0", "0"]
