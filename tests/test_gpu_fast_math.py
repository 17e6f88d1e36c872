"""The range-free division, reciprocal and square root of the shading kernels against the IEEE operators, and the
dielectric sample built on them, alone and two at a time, against the one built on the operators, bit for bit."""
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
__device__ float unit(uint64_t x) { return (float)(mixed(x) >> 8) * 0x1p-24f; }

// every significand, every exponent of the stated ranges
__global__ void one_argument(unsigned long long* bad) {
    const uint32_t m = blockIdx.x * blockDim.x + threadIdx.x;
    for (int e = -120; e <= 120; ++e) {
        const float b = make(e, m);
        if (!same(rcp_in_range(b), 1.0f / b) || !same(rcp_in_range(-b), 1.0f / -b)) atomicAdd(bad, 1ull);
    }
    for (int e = -96; e <= 126; ++e)
        if (!same(sqrt_in_range(make(e, m)), sqrtf(make(e, m)))) atomicAdd(bad + 1, 1ull);
    for (int e = -96; e <= 100; ++e)
        if (!same(rcp_in_range(sqrt_in_range(make(e, m))), 1.0f / sqrtf(make(e, m)))) atomicAdd(bad + 2, 1ull);
}

__device__ bool agree(float a, float b) { return same(a, b) || (a != a && b != b); }

// the functions that take any argument, on every float
__global__ void any_argument(unsigned long long* bad) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    for (uint32_t k = 0; k < 256; ++k) {
        const float b = __uint_as_float(i * 256u + k);
        if (!agree(rcp(b), 1.0f / b)) atomicAdd(bad + 3, 1ull);
        if (!agree(ptd::sqrt_(b), sqrtf(b)) || !agree(rsqrt_(b), 1.0f / sqrtf(b))) atomicAdd(bad + 3, 1ull);
        if (!agree(acos_(b), ptm::acosf_(b))) atomicAdd(bad + 3, 1ull);
        const float turn = fabsf(b);
        float s, c, s1, c1;
        if (turn <= kTwoPi) {
            sincos_turn(turn, &s, &c);
            ptm::sincosf_(turn, &s1, &c1);
            if (!same(s, s1) || !same(c, c1)) atomicAdd(bad + 3, 1ull);
        }
        // arc tangents: against a second argument of every kind
        const uint32_t r = mixed(((uint64_t)i << 8) + k);
        const float others[6] = {__uint_as_float(r), b, 0.0f, -0.0f, __uint_as_float(0x7f800000u), (float)(r >> 8) * 0x1p-23f - 1.0f};
        for (float o : others) {
            if (!agree(atan2_(b, o), ptm::atan2f_(b, o)) || !agree(atan2_(o, b), ptm::atan2f_(o, b)) ||
                !agree(atan2_(b, -o), ptm::atan2f_(b, -o)))
                atomicAdd(bad + 3, 1ull);
        }
    }
}

// bytes as unorm, the sky's column over its width
__global__ void constants(unsigned long long* bad) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < 256u && !same(div_by((float)i, 255.0f, 1.0f / 255.0f), (float)i / 255.0f)) atomicAdd(bad + 4, 1ull);
    const uint32_t width = 1u + mixed(i) % 16384u, column = mixed(~i) % width;
    const float a = (float)column + unit(i), w = (float)width;
    if (!same(div_by(a, w, 1.0f / w), a / w)) atomicAdd(bad + 4, 1ull);
}

// quotients: random significands, and the hard ones (divisors of ones, numerators next to the divisor or to 1 or 2)
__global__ void quotients(unsigned long long* bad) {
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (uint32_t i = 0; i < 1024u; ++i) {
        const uint64_t k = t * 1024u + i;
        uint32_t a = mixed(2 * k) & 0x7fffffu, b = mixed(2 * k + 1) & 0x7fffffu;
        const uint32_t kind = i & 7u, r = mixed(~k);
        if (kind == 4u) b = 0x7fffffu - (r & 7u);
        if (kind == 5u) a = r & 63u;
        if (kind == 6u) a = 0x7fffffu - (r & 63u);
        if (kind == 7u) a = (b + (r % 9u) - 4u) & 0x7fffffu;
        const float y = make((int)(r >> 8) % 61, b), x = make((int)(r >> 16) % 61 - 30, a);
        if (!same(div_in_range(x, y), x / y) || !same(div_in_range(-x, y), -x / y) || !same(div_in_range(x, -y), x / -y)) atomicAdd(bad + 4, 1ull);
        if (!same(div_in_range(0.0f, y), 0.0f) || !same(div_in_range(-0.0f, y), -0.0f)) atomicAdd(bad + 4, 1ull);
    }
}

__global__ void samples(unsigned long long* bad, unsigned long long* count) {
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned used = 0, redone = 0;
    for (uint32_t i = 0; i < 256u; ++i) {
        const uint64_t k = (t * 256u + i) * 16u;
        DielectricTerms d;
        const float rough = unit(k), aniso = (i & 3u) ? 0.0f : unit(k + 1);
        d.alpha = alpha_anisotropic((i & 12u) ? rough : 0.0f, aniso);
        // from grazing views to the normal itself
        const float cz = (i & 48u) ? unit(k + 2) : 1e-4f * unit(k + 2) + ((i & 1u) ? 0.0f : 0.9999f);
        const float sz = sqrtf(saturate(1.0f - cz * cz)), ph = kTwoPi * unit(k + 3);
        d.wo = (i & 192u) ? mk(sz * cosf(ph), sz * sinf(ph), cz) : mk(0.0f, 0.0f, 1.0f);
        d.ww = vndf_view(d.wo, d.alpha);
        d.ww1 = 1.0f + d.ww.z;
        d.ior = (i & 2u) ? 1.0f + 2.0f * unit(k + 4) : ((i & 1u) ? 1.5f : 0.5f + unit(k + 4));
        d.ior2 = d.ior * d.ior;
        d.rcp_ior2 = 1.0f / d.ior2;
        d.ax2 = d.alpha.x * d.alpha.x;
        d.ay2 = d.alpha.y * d.alpha.y;
        d.opl = 1.0f + ggx_lambda(d.wo, d.alpha);
        if (!dielectric_fast(d)) continue;
        uint32_t s = mixed(k + 5);
        const float r1 = rand_next(s), tpr = kTwoPi * rand_next(s);
        bool redo = false;
        const float fast = dielectric_sample_fast(d, r1, tpr, &redo), want = dielectric_sample(d, r1, tpr);
        used += 1u;
        redone += redo;
        if (!redo && !agree(fast, want)) atomicAdd(bad + 5, 1ull);
        // two samples packed: this one and the next, in either place
        const float r2 = rand_next(s), tpr2 = kTwoPi * rand_next(s);
        bool redo2 = false, pair_redo = false, swapped_redo = false;
        float a, b, c, e;
        const float fast2 = dielectric_sample_fast(d, r2, tpr2, &redo2);
        dielectric_pair_fast(d, r1, tpr, r2, tpr2, &a, &b, &pair_redo);
        dielectric_pair_fast(d, r2, tpr2, r1, tpr, &c, &e, &swapped_redo);
        if (pair_redo != (redo || redo2) || swapped_redo != pair_redo) atomicAdd(bad + 5, 1ull);
        if (!pair_redo && (!agree(a, fast) || !agree(b, fast2) || !agree(c, fast2) || !agree(e, fast))) atomicAdd(bad + 5, 1ull);
    }
    atomicAdd(count, (unsigned long long)used);
    atomicAdd(count + 1, (unsigned long long)redone);
}

int main() {
    unsigned long long *bad, h[8] = {0};
    if (cudaMalloc(&bad, 64) != cudaSuccess || cudaMemset(bad, 0, 64) != cudaSuccess) return 2;
    one_argument<<<(1 << 23) / 256, 256>>>(bad);
    any_argument<<<(1 << 24) / 256, 256>>>(bad);
    constants<<<1 << 14, 256>>>(bad);
    quotients<<<1 << 11, 256>>>(bad);
    samples<<<1 << 10, 256>>>(bad, bad + 6);
    if (cudaMemcpy(h, bad, 64, cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
    for (int i = 0; i < 8; ++i) printf("%llu ", h[i]);
    return 0;
}
"""


def test_range_free_operations_are_correctly_rounded(tmp_path):
    src, exe = tmp_path / "fast_math.cu", tmp_path / "fast_math"
    src.write_text(SOURCE)
    subprocess.run([build.NVCC, *build.NVCC_FLAGS, f"-I{build.CSRC}", f"-I{build.INCLUDE}", str(src), "-o", str(exe)],
                   check=True, capture_output=True, timeout=300)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=120).stdout
    *bad, used, redone = (int(v) for v in out.split())
    assert bad == [0] * 6
    assert used > 50_000_000 and redone < used // 1000
