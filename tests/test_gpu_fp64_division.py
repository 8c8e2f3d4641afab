"""The FP64 reciprocal, quotient, square root and van Leer limiter of the kernels against the device's own division and
square root (GPU required).  Each ends in a residual step from an approximation within 1 ulp, which rounds correctly
(Markstein): equal at ordinary exponents; at most 1 ulp apart over any bit patterns, where a residual can underflow; the same infinities, zeros and NaN."""
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
#include "common.cuh"
constexpr int F = 4;
__global__ void probe(const double* x, const double* y, double* o, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double a = x[i], b = y[i], p = a * b, num = p > 0 ? p : 0.0, st = num / (a + b);
    double* r = o + 2 * F * (size_t)i;
    r[0] = img::recip(b);                              r[1] = 1.0 / b;
    r[2] = img::quotient(a, b);                        r[3] = a / b;
    r[4] = img::sqrt_goldschmidt(fabs(b));             r[5] = sqrt(fabs(b));
    r[6] = img::limiter_corr_t<img::LIM_VANLEER>(a, b);     r[7] = isnan(st) ? 0.0 : st;
}
static double off(double a, double b) {   // in units of the last place of b; 0 for equal specials
    if (std::isnan(b)) return std::isnan(a) ? 0 : 1e9;
    if (a == b) return 0;
    if (!std::isfinite(a) || !std::isfinite(b)) return 1e9;
    return std::fabs(a - b) / (std::nextafter(std::fabs(b), INFINITY) - std::fabs(b));
}
int main() {
    const double sp[] = {0.0, -0.0, INFINITY, -INFINITY, NAN, 5e-324, -2.2250738585072014e-308, 1.7976931348623157e308, 1.0, -1.0, 1e-200, 1e200};
    std::vector<double> x, y;
    for (double a : sp) for (double b : sp) { x.push_back(a); y.push_back(b); }
    const int nsp = (int)x.size(), n = nsp + (1 << 21);
    unsigned long long z = 88172645463325252ull;
    auto next = [&](bool any) {
        z ^= z << 13; z ^= z >> 7; z ^= z << 17;
        unsigned long long b = z;
        if (!any) {   // ordinary exponents; every fourth mantissa within 64 of all zeros or all ones
            if (z >> 62 == 0) b = (z & 0x8000000000000000ull) | ((z & 64) ? 0x000fffffffffffffull - (z & 63) : (z & 63));
            b = (b & 0x800fffffffffffffull) | ((unsigned long long)(1023 - 20 + (z >> 7) % 41) << 52);
        }
        double v;
        std::memcpy(&v, &b, 8);
        return v;
    };
    for (int i = nsp; i < n; ++i) { x.push_back(next(i & 1)); y.push_back(next(i & 1)); }
    double *d, *o;
    cudaMalloc(&d, 2 * (size_t)n * 8);
    cudaMalloc(&o, 2 * F * (size_t)n * 8);
    cudaMemcpy(d, x.data(), n * 8, cudaMemcpyHostToDevice);
    cudaMemcpy(d + n, y.data(), n * 8, cudaMemcpyHostToDevice);
    probe<<<(n + 255) / 256, 256>>>(d, d + n, o, n);
    std::vector<double> h(2 * F * (size_t)n);
    if (cudaMemcpy(h.data(), o, h.size() * 8, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    double worst[F] = {}, ordinary[F] = {};
    for (int i = 0; i < n; ++i)
        for (int f = 0; f < F; ++f) {
            if (f == 3 && !(std::fabs(x[i] + y[i]) < 1e300)) continue;   // sums the reciprocal's estimate would flush
            const double e = off(h[2 * F * (size_t)i + 2 * f], h[2 * F * (size_t)i + 2 * f + 1]);
            worst[f] = std::fmax(worst[f], e);
            if (i >= nsp && !(i & 1)) ordinary[f] = std::fmax(ordinary[f], e);
        }
    int bad = 0;
    for (int f = 0; f < F; ++f) {
        std::printf("%d: any %g ulp, ordinary %g ulp\n", f, worst[f], ordinary[f]);
        bad |= !(worst[f] <= 1.0) || ordinary[f] != 0;
    }
    return bad;
}
"""


def test_division_and_square_root_round_correctly(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    src = tmp_path / "probe.cu"
    src.write_text(PROGRAM)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17", "-I",
                    os.path.join(ROOT, "imogen_b200", "csrc"), str(src), "-o", str(tmp_path / "probe")], check=True, capture_output=True)
    r = subprocess.run([str(tmp_path / "probe")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
