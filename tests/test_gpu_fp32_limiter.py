"""The FP32 limiters of the segment and window kernels' lanes against those of the pencil-tile kernels (GPU required), bit
for bit: pairs of fluxes' differences over all signs, exponents where the product or the sum overflows or underflows,
zeros, infinities and NaN.  A NaN quotient counts as no correction (vanleerLimiter.m:11)."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>
#include "lanes.cuh"
using namespace img;
template <int LIM>
__device__ void three(float a, float b, float* r) {
    r[0] = limiter_corr_t<LIM>(a, b);
    r[1] = v_limit<LIM>(a, b);
    float x, y;
    v_limit<LIM>(F2(a, b), F2(b, a)).get(x, y);   // (x: a, b)
    r[2] = x;
}
__global__ void probe(const float* x, const float* y, float* o, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    three<LIM_VANLEER>(x[i], y[i], o + 9 * (size_t)i);
    three<LIM_SUPERBEE>(x[i], y[i], o + 9 * (size_t)i + 3);
    three<LIM_MINMOD>(x[i], y[i], o + 9 * (size_t)i + 6);
}
int main() {
    const float sp[] = {0.f, -0.f, INFINITY, -INFINITY, NAN, 1e-45f, -1e-38f, 3.4028235e38f, -3.4028235e38f, 2e38f, 1e38f, 1e20f, 2e19f, -1e20f, 1e-20f, 1e-23f, 1.f, -1.f};
    std::vector<float> x, y;
    for (float a : sp) for (float b : sp) { x.push_back(a); y.push_back(b); }
    unsigned long long z = 88172645463325252ull;
    for (int i = 0; i < 1 << 20; ++i) {   // any bit patterns
        z ^= z << 13; z ^= z >> 7; z ^= z << 17;
        const unsigned a = (unsigned)z, b = (unsigned)(z >> 32);
        float u, v;
        std::memcpy(&u, &a, 4);
        std::memcpy(&v, &b, 4);
        x.push_back(u); y.push_back(v);
    }
    const int n = (int)x.size();
    float *d, *o;
    cudaMalloc(&d, 2 * (size_t)n * 4);
    cudaMalloc(&o, 9 * (size_t)n * 4);
    cudaMemcpy(d, x.data(), n * 4, cudaMemcpyHostToDevice);
    cudaMemcpy(d + n, y.data(), n * 4, cudaMemcpyHostToDevice);
    probe<<<(n + 255) / 256, 256>>>(d, d + n, o, n);
    std::vector<float> h(9 * (size_t)n);
    if (cudaMemcpy(h.data(), o, h.size() * 4, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    int bad = 0;
    for (int i = 0; i < n; ++i)
        for (int l = 0; l < 3; ++l)
            for (int f = 1; f < 3; ++f) {
                const float e = h[9 * (size_t)i + 3 * l], g = h[9 * (size_t)i + 3 * l + f];
                if (!(e == g || (std::isnan(e) && std::isnan(g))) && bad++ < 20)
                    std::printf("limiter %d form %d of %g and %g: %g, not %g\n", l, f, x[i], y[i], g, e);
            }
    std::printf("%d differ\n", bad);
    return bad != 0;
}
"""


def test_lanes_limit_as_the_tile_kernels_do(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    src = tmp_path / "probe.cu"
    src.write_text(PROGRAM)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17", "-I",
                    os.path.join(ROOT, "imogen_b200", "csrc"), str(src), "-o", str(tmp_path / "probe")], check=True, capture_output=True)
    r = subprocess.run([str(tmp_path / "probe")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
