"""The range-free quotients, alone and two at a time, against the operator over the whole range that they are stated
for: divisors of 2^-60 .. 2^60 of either sign, numerators and quotients of 2^-100 .. 2^100, zero numerators; and the
packed reciprocal and root.  Random significands and the hard ones (divisors near the next power of two, numerators
next to the divisor, to 1 or to 2), exponents from other bits than the significands.  Bit for bit."""
import subprocess

import pytest

from pathtracer import build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include <cstdio>
#include "pt_device.cuh"
using namespace ptd;

__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }
__device__ float make(int exponent, uint32_t significand) { return __uint_as_float(((uint32_t)(exponent + 127) << 23) | significand); }
__device__ uint32_t mixed(uint64_t x) {
    x ^= x >> 33; x *= 0xff51afd7ed558ccdull; x ^= x >> 33; x *= 0xc4ceb9fe1a85ec53ull; x ^= x >> 33;
    return (uint32_t)x;
}
__device__ bool same(Two t, float a, float b) { return same(first(t), a) && same(second(t), b); }

// bad: 0 one quotient, 1 two, 2 zero numerators, 3 packed reciprocals and roots; 4 counts the quotients compared
__global__ void quotients(unsigned long long* bad) {
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned used = 0;
    for (uint32_t i = 0; i < 512u; ++i) {
        const uint64_t k = (t * 512u + i) * 8u;
        float x[2], y[2];
        for (int j = 0; j < 2; ++j) {
            uint32_t a = mixed(k + 4 * j) & 0x7fffffu, b = mixed(k + 4 * j + 1) & 0x7fffffu;
            const uint32_t r = mixed(k + 4 * j + 2), e = mixed(k + 4 * j + 3), kind = r & 7u;
            if (kind == 4u) b = 0x7fffffu - ((r >> 3) & 7u);
            if (kind == 5u) a = (r >> 3) & 63u;
            if (kind == 6u) a = 0x7fffffu - ((r >> 3) & 63u);
            if (kind == 7u) a = (b + ((r >> 3) % 9u) - 4u) & 0x7fffffu;
            const int eb = (int)(e & 0xffffu) % 121 - 60;
            // a quotient is at least 2^(ea - eb - 1) and below 2^(ea - eb + 1)
            const int lo = max(-100, eb - 99), hi = min(99, eb + 98);
            const int ea = lo + (int)((e >> 16) % (uint32_t)(hi - lo + 1));
            x[j] = make(ea, a) * ((r >> 30) & 1u ? -1.0f : 1.0f);
            y[j] = make(eb, b) * ((r >> 31) & 1u ? -1.0f : 1.0f);
            const float q = x[j] / y[j];
            if (!same(div_in_range(x[j], y[j]), q) || !same(div_by(x[j], y[j], 1.0f / y[j]), q)) atomicAdd(bad, 1ull);
            used += 1u;
            const float z = fabsf(y[j]);
            if (!same(div_in_range(0.0f, z), 0.0f) || !same(div_in_range(-0.0f, z), -0.0f) || !same(div_by(0.0f, z, 1.0f / z), 0.0f) ||
                !same(div_in_range(two(0.0f), two(z)), 0.0f, 0.0f))
                atomicAdd(bad + 2, 1ull);
        }
        const float q0 = x[0] / y[0], q1 = x[1] / y[1];
        for (int s = 0; s < 2; ++s) {
            const Two a = s ? two(x[1], x[0]) : two(x[0], x[1]), b = s ? two(y[1], y[0]) : two(y[0], y[1]);
            const float p = s ? q1 : q0, q = s ? q0 : q1;
            const Two one = two(1.0f / first(b), 1.0f / second(b));
            if (!same(div_in_range(a, b), p, q) || !same(div_by(a, negated(b), one), p, q)) atomicAdd(bad + 1, 1ull);
            const float u = fabsf(first(b)), v = fabsf(second(b));
            if (!same(rcp_in_range(b), first(one), second(one)) || !same(sqrt_in_range(two(u, v)), sqrtf(u), sqrtf(v)))
                atomicAdd(bad + 3, 1ull);
        }
    }
    atomicAdd(bad + 4, (unsigned long long)used);
}

int main() {
    unsigned long long *bad, h[5] = {0};
    if (cudaMalloc(&bad, 64) != cudaSuccess || cudaMemset(bad, 0, 64) != cudaSuccess) return 2;
    quotients<<<1 << 12, 256>>>(bad);
    if (cudaMemcpy(h, bad, 40, cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
    for (unsigned long long v : h) printf("%llu ", v);
    return 0;
}
"""


def test_quotients_are_correctly_rounded_over_their_range(tmp_path):
    src, exe = tmp_path / "quotients.cu", tmp_path / "quotients"
    src.write_text(SOURCE)
    subprocess.run([build.NVCC, *build.NVCC_FLAGS, f"-I{build.CSRC}", f"-I{build.INCLUDE}", str(src), "-o", str(exe)],
                   check=True, capture_output=True, timeout=300)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=120).stdout
    *bad, used = (int(v) for v in out.split())
    assert used > 1_000_000_000
    assert bad == [0] * 4
