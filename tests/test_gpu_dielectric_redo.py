"""The dielectric estimate of a hit in which a sample leaves the range of the unchecked operations, so that all 16 are
taken again with checked ones: its sum, the random state after it and the random draws it records, alone and with the
hit's lanes sharing the samples, against the checked samples in order.  The hits are searched for (a sampled direction
in the surface's plane, one hit in millions), and made (views of length 2^-40, every sample of which leaves the range)."""
import subprocess

import pytest

from pathtracer import build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include <cstdio>
#include "pt_device.cuh"
using namespace ptd;

__device__ bool agree(float a, float b) { return __float_as_uint(a) == __float_as_uint(b) || (a != a && b != b); }
__device__ uint32_t mixed(uint64_t x) {
    x ^= x >> 33; x *= 0xff51afd7ed558ccdull; x ^= x >> 33; x *= 0xc4ceb9fe1a85ec53ull; x ^= x >> 33;
    return (uint32_t)x;
}
__device__ float unit(uint64_t x) { return (float)(mixed(x) >> 8) * 0x1p-24f; }

struct Hit {
    DielectricTerms t;
    uint32_t seed;
};
// hit number k: a view anywhere above the surface, any roughness; made: a view of length 2^-40
__device__ Hit hit(uint64_t k, bool made) {
    Hit h;
    k *= 16u;
    h.t.alpha = alpha_anisotropic(0.05f + 0.95f * unit(k), unit(k + 1));
    const float cz = 1.0f - unit(k + 2), sz = sqrtf(saturate(1.0f - cz * cz)), ph = kTwoPi * unit(k + 3);
    h.t.wo = mk(sz * cosf(ph), sz * sinf(ph), cz) * (made ? 0x1p-40f : 1.0f);
    h.t.ww = vndf_view(h.t.wo, h.t.alpha);
    h.t.ww1 = 1.0f + h.t.ww.z;
    h.t.ior = 1.0f + 2.0f * unit(k + 4);
    h.t.ior2 = h.t.ior * h.t.ior;
    h.t.rcp_ior2 = 1.0f / h.t.ior2;
    h.t.ax2 = h.t.alpha.x * h.t.alpha.x;
    h.t.ay2 = h.t.alpha.y * h.t.alpha.y;
    h.t.opl = 1.0f + ggx_lambda(h.t.wo, h.t.alpha);
    h.seed = mixed(k + 5) | 1u;
    return h;
}

constexpr unsigned kMost = 4096;
__global__ void search(unsigned* found, unsigned long long* which) {
    const uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const Hit h = hit(k, false);
    if (!dielectric_fast(h.t)) return;
    bool redo = false;
    uint32_t s = h.seed;
    for (int i = 0; i < 8; ++i) {
        float a, b;
        const float ra = rand_next(s), ta = kTwoPi * rand_next(s), rb = rand_next(s), tb = kTwoPi * rand_next(s);
        dielectric_pair_fast(h.t, ra, ta, rb, tb, &a, &b, &redo);
    }
    if (!redo) return;
    const unsigned at = atomicAdd(found, 1u);
    if (at < kMost) which[at] = k;
}

// one warp per hit; bad: 0 the sum, 1 the random state, 2 the draws, 3 a made hit that stays in range
__global__ void check(unsigned n, const unsigned long long* which, bool made, unsigned* bad) {
    const unsigned w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31u;
    if (w >= n) return;
    const Hit h = hit(made ? w : which[w], made);
    uint32_t s = h.seed;
    float sum = 0.0f;
    bool redo = false;
    for (int i = 0; i < 16; ++i) {
        const float r1 = rand_next(s), tpr = kTwoPi * rand_next(s);
        sum += dielectric_sample(h.t, r1, tpr);
        dielectric_sample_fast(h.t, r1, tpr, &redo);
    }
    if (!redo) atomicAdd(bad + 3, 1u);
    const f3 want = mk(0.9f, 0.5f, 0.25f) * sum / 16.0f;
    const auto compare = [&](f3 got, uint32_t state) {
        if (!agree(got.x, want.x) || !agree(got.y, want.y) || !agree(got.z, want.z)) atomicAdd(bad, 1u);
        if (state != s) atomicAdd(bad + 1, 1u);
    };
    Counters c{};
    Rng<true> counted;
    counted.s = h.seed;
    counted.rec.c = &c;
    compare(estimate_e_dielectric<true, false>(h.t.wo, h.t.opl, h.t.alpha, h.t.ior, mk(0.9f, 0.5f, 0.25f), counted, Spread()), counted.s);
    if (c.rand_draws != 32u) atomicAdd(bad + 2, 1u);
    for (uint32_t log2 = 0; log2 <= 4; ++log2) {
        Rng<false> plain;
        plain.s = h.seed;
        Spread spread;
        spread.log2 = log2;
        spread.index = lane & ((1u << log2) - 1u);
        spread.mask = ((1u << (1u << log2)) - 1u) << (lane - spread.index);
        const f3 e = estimate_e_dielectric<false, true>(h.t.wo, h.t.opl, h.t.alpha, h.t.ior, mk(0.9f, 0.5f, 0.25f), plain, spread);
        compare(e, plain.s);
        __syncwarp();
    }
}

int main() {
    unsigned *count, h[5] = {0};
    unsigned long long* which;
    if (cudaMalloc(&count, 32) != cudaSuccess || cudaMalloc(&which, kMost * 8) != cudaSuccess) return 2;
    if (cudaMemset(count, 0, 32) != cudaSuccess || cudaMemset(which, 0, kMost * 8) != cudaSuccess) return 2;
    search<<<1 << 21, 256>>>(count, which);
    if (cudaMemcpy(h, count, 4, cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
    const unsigned n = h[0] < kMost ? h[0] : kMost;
    if (n) check<<<(n + 3) / 4, 128>>>(n, which, false, count + 1);
    check<<<16, 128>>>(64, which, true, count + 1);
    if (cudaMemcpy(h, count, 20, cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
    for (unsigned v : h) printf("%u ", v);
    return 0;
}
"""


def test_a_redone_estimate_equals_the_checked_samples(tmp_path):
    src, exe = tmp_path / "redo.cu", tmp_path / "redo"
    src.write_text(SOURCE)
    subprocess.run([build.NVCC, *build.NVCC_FLAGS, f"-I{build.CSRC}", f"-I{build.INCLUDE}", str(src), "-o", str(exe)],
                   check=True, capture_output=True, timeout=300)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=120).stdout
    found, *bad = (int(v) for v in out.split())
    print("searched hits with a redone estimate:", found)
    assert found > 0
    assert bad == [0] * 4
