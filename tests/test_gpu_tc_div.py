"""The division of the grouped GEMM's task end (tc_div of csrc/gemm_tc.cuh) against the compiler's, bit for bit: every divisor of a
binade with numerators of random bits, gates with their own denominators, and the ends of the range outside of which the caller
divides again."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include "gemm_tc.cuh"
// [0] quotients, [1] of these in range, [2] in range and not the compiler's, [3] range decided otherwise than stated
__device__ unsigned long long c_count[4];
__device__ void check(float a, float d, unsigned long long (&n)[4]) {
    bool odd = false;
    const float q = tc_div(a, d, odd), want = a / d;
    const bool in = d < 1e10f && fabsf(a) > 1e-20f && fabsf(a) < 1e20f;
    n[0]++;
    if (odd == in) n[3]++;
    if (!odd) { n[1]++; if (__float_as_uint(q) != __float_as_uint(want)) n[2]++; }
}
__device__ uint32_t mix(uint32_t x) { x ^= x >> 16; x *= 0x7feb352du; x ^= x >> 15; x *= 0x846ca68bu; return x ^ (x >> 16); }
__global__ void k_check(int per) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;           // 2^23 threads: the mantissa of the divisor
    unsigned long long n[4] = {0, 0, 0, 0};
    uint32_t r = mix(i + 1);
    for (int k = 0; k < per; k++) {
        r = mix(r + k);
        const float any = __uint_as_float(r), d = __uint_as_float((127u + (k % 34)) << 23 | i);      // 1 to 2^34
        check(any, d, n);                                               // any bits, infinities and NaN among them
        const uint32_t m = mix(r);
        check(__uint_as_float((m & 0x80000000u) | (96u + (m >> 23) % 64u) << 23 | (m & 0x7fffffu)), d, n);     // 2^-31 to 2^33
        const float g = __uint_as_float((m & 0x80000000u) | (100u + (m >> 23) % 34u) << 23 | (r & 0x7fffffu)); // a gate, 2^-27 to 2^6
        check(g, 1.0f + expf(-g), n);
    }
    if (i < 4096) {                                                     // around the ends of the range, both signs
        const float ends[] = {1e-20f, 1e20f, 0.f, 1.17549435e-38f}, div[] = {1e10f, 1.f, 3.4028235e38f};
        for (int s = 0; s < 2; s++)
            for (float e : ends)
                for (float d : div) {
                    const float a = __uint_as_float(__float_as_uint(e) + i % 64u - (e > 0.f ? 32u : 0u)), dd = __uint_as_float(__float_as_uint(d) + i / 64u - (d > 1.f ? 32u : 0u));
                    check(s ? -a : a, dd, n);
                }
        check(1.f, __uint_as_float(0x7f800000u), n); check(1.f, __uint_as_float(0x7fc00000u), n);
    }
    for (int k = 0; k < 4; k++) atomicAdd(c_count + k, n[k]);
}
extern "C" int run(int per, unsigned long long *out) {
    k_check<<<(1 << 23) / 256, 256>>>(per);
    return cudaMemcpyFromSymbol(out, c_count, 4 * sizeof(*out)) == cudaSuccess;
}
"""


def test_every_bit_of_the_quotient(tmp_path):
    from colibri_b200 import build
    if not shutil.which(build.NVCC):
        pytest.skip("no nvcc")
    src, lib = tmp_path / "div.cu", tmp_path / "div.so"
    src.write_text(SOURCE)
    env = {k: v for k, v in os.environ.items() if k not in ("CC", "CXX")}
    subprocess.check_call([build.NVCC] + build.FLAGS + ["-I", build.CSRC, "-o", str(lib), str(src), "-ccbin", "/usr/bin/g++"], env=env)
    n = (C.c_ulonglong * 4)()
    assert C.CDLL(str(lib)).run(34, n) == 1
    assert n[0] > 8e8 and n[1] > 5e8, list(n)
    assert n[2] == 0 and n[3] == 0, list(n)
