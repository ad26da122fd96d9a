"""The walk's division-free quotients (device_common.cuh) against the plain operations, bit for bit: the
corrected reciprocal for every significand, quotients by a shared divisor and packed in pairs, the
packed logarithm, and zero numerators of both signs."""
from __future__ import annotations

import os
import subprocess

import pytest

from wobtoolbox_gb300 import build as B

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include "device_common.cuh"
#include <cstdio>
using namespace wobgb;

__device__ unsigned long long bad[4];

__device__ __forceinline__ uint32_t bits(float x) { return __float_as_uint(x); }
// sign and significand of h, exponent 2^-60 .. 2^59 by e
__device__ __forceinline__ float mid(uint32_t h, uint32_t e, bool sign) {
    return __uint_as_float((h & 0x007fffffu) | ((67u + e % 120u) << 23) | (sign ? h & 0x80000000u : 0u));
}
__device__ __forceinline__ float wide(uint32_t h, uint32_t e) { return mid(h, e, true); }

// every significand, exponents across the range
__global__ void reciprocals() {
    const uint32_t m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= (1u << 23)) return;
    for (uint32_t e = 0; e < 120; e += 17) {
        const float b = mid(m, e, false);
        if (bits(shared_divisor(b).y) != bits(1.0f / b)) atomicAdd(bad, 1ull);
    }
}
__global__ void quotients(uint64_t n, uint64_t neg_zero) {
    const F2 z{neg_zero};
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint4 h = philox4x32_10(make_uint4((uint32_t)i, (uint32_t)(i >> 32), 1u, 2u), 3u, 4u);
        const uint4 g = philox4x32_10(make_uint4((uint32_t)i, (uint32_t)(i >> 32), 5u, 2u), 3u, 4u);
        const float a0 = wide(h.x, g.x), a1 = wide(h.y, g.y), b0 = mid(h.z, g.z, false), b1 = mid(h.w, g.w, false);
        const SharedDivisor d = shared_divisor(b0);
        if (bits(shared_quotient(a0, d)) != bits(a0 / b0) || bits(shared_quotient(a1, d)) != bits(a1 / b0)) atomicAdd(bad + 1, 1ull);
        const F2 q = f2quotient(f2(a0, a1), f2(b0, b1), z);
        if (bits(f2lo(q)) != bits(a0 / b0) || bits(f2hi(q)) != bits(a1 / b1)) atomicAdd(bad + 2, 1ull);
        const F2 l = f2log(f2(b0, b1), z);
        if (bits(f2lo(l)) != bits(log_own(b0)) || bits(f2hi(l)) != bits(log_own(b1))) atomicAdd(bad + 2, 1ull);
        // zero numerators, alone and in a vector whose other component makes the length
        for (int s = 0; s < 2; s++) {
            const float zero = s ? -0.0f : 0.0f;
            if (bits(shared_quotient(zero, d)) != bits(zero / b0)) atomicAdd(bad + 3, 1ull);
            const V<2> v = vnormalized(V<2>{{zero, a0}}), w = vdiv(V<2>{{zero, a0}}, sqrtf(vsqnorm(V<2>{{zero, a0}})));
            if (bits(v.v[0]) != bits(w.v[0]) || bits(v.v[1]) != bits(w.v[1])) atomicAdd(bad + 3, 1ull);
        }
    }
}
int main() {
    reciprocals<<<(1 << 23) / 256, 256>>>();
    quotients<<<1216, 256>>>(1ull << 28, f2_neg_zero);
    unsigned long long h[4] = {~0ull, ~0ull, ~0ull, ~0ull};
    if (cudaMemcpyFromSymbol(h, bad, sizeof h) != cudaSuccess) return 1;
    printf("%llu %llu %llu %llu\n", h[0], h[1], h[2], h[3]);
    return 0;
}
"""


@pytest.fixture(scope="module")
def mismatches(cuda, tmp_path_factory):
    d = tmp_path_factory.mktemp("quotients")
    src, exe = d / "q.cu", d / "q"
    src.write_text(PROGRAM)
    subprocess.run([B.nvcc_path()] + B.cu_flags() + ["-I", B.CSRC, str(src), "-o", str(exe)], check=True,
                   capture_output=True, text=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=120,
                         env=dict(os.environ)).stdout
    return [int(x) for x in out.split()]


def test_reciprocals_of_every_significand(mismatches):
    assert mismatches[0] == 0


def test_quotients_and_logarithms(mismatches):
    assert mismatches[1] == 0 and mismatches[2] == 0


def test_signed_zero_numerators(mismatches):
    assert mismatches[3] == 0
