"""Segment fluid and window magnet kernels where they can go wrong (GPU required): pencils of every remainder of
the cells per thread along every direction, last segments of one cell, pencils shorter than two segments, CTAs
with idle threads, circ, const and fade ends and mixtures of them, against the C++ oracle.

Relative L1 per variable after 4 iterations: FP64 1e-11, the mixed form 2e-5 (the tolerances of the other
oracle comparisons of these kernels)."""
import os
import shutil
import subprocess

import pytest

from imogen_b200 import ImogenBatch, ImogenRun
from tests.parity import errors, make_pair, smooth_state

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
TOL = {"fp64": 1e-11, "mixed": 2e-5}


def _settings(grid, bc, magnet, limiter=("vanleer", "minmod", "superbee")):
    return dict(grid=grid, dgrid=(1.0 / max(grid),) * 3, gamma=5 / 3, cfl=0.35, bc=bc, limiter=limiter, magnet=magnet,
                time_max=1e5, iter_max=10 ** 6)


def _compare(settings, state, precision, tilings=(), iters=4):
    o, g = make_pair(settings, state, precision=precision)
    for kind, dim, t in tilings:
        g.set_tiling(dim, t, kind=kind)
    swept = [d for d in (1, 2, 3) if settings["grid"][d - 1] >= 3]
    assert all(g.tiling("fluid")[d][6] for d in swept), g.tiling("fluid")
    o.run(iters)
    g.run(iters)
    e = errors(g.state(), o.state())
    g.close()
    bad = {k: v for k, v in e.items() if not v <= TOL[precision]}
    assert not bad, bad


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("bc", ["circ", "const"])
@pytest.mark.parametrize("grid", [(5, 6, 7), (9, 13, 10), (21, 22, 23), (33, 37, 12), (70, 81, 1)])
def test_every_remainder_along_every_direction(grid, bc, precision):
    _compare(_settings(grid, bc, True), smooth_state(grid, seed=3, mhd=True), precision)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("cells", [2, 4])
@pytest.mark.parametrize("magnet", [False, True])
@pytest.mark.parametrize("grid,bc", [((20, 21, 1), "fade"), ((41, 22, 23), "fade"), ((64, 27, 1), {"x": ("fade", "const"), "y": ("circ", "fade")}),
                                     ((35, 32, 1), {"x": ("const", "fade"), "y": ("fade", "circ")})])
def test_fade_ends(grid, bc, magnet, cells, precision):
    """Fade ends on one or both sides, at the shortest pencils that take them (20 cells, where the damping of
    both ends overlaps) and ragged ones."""
    if not isinstance(bc, str):
        bc = {**bc, "z": "circ"}
    til = []
    for d in (1, 2, 3):
        n = grid[d - 1]
        if n >= 3:
            s = -(-n // cells)
            wb = next(w for w in ((1, 2, 4, 8, 16, 32) if d == 1 else (4, 8, 16, 32)) if w * s >= 64 or w == 32)
            til.append(("fluid", d, (wb, s, 1, -(-wb * s // 32) * 32, cells, 1, 1)))
    _compare(_settings(grid, bc, magnet), smooth_state(grid, seed=8, mhd=magnet), precision, til)


@pytest.mark.parametrize("cells", [2, 4, 8])
@pytest.mark.parametrize("n", [64, 65, 66, 67, 73])
def test_mixed_cells_per_thread(n, cells):
    grid = (n, 24, 1)
    s = -(-n // cells)
    wb = next(w for w in (1, 2, 4, 8, 16, 32) if w * s >= 64)
    t = (wb, s, 1, -(-wb * s // 32) * 32, cells, 1, 1)
    _compare(_settings(grid, "circ", True), smooth_state(grid, seed=5, mhd=True), "mixed",
             [("fluid", 1, t), ("magnet", 1, t)])


def test_fade_members_of_a_batch_equal_their_runs_alone():
    grids = [(40, 33, 1), (52, 41, 1), (64, 64, 1)]
    alone, together = [], []
    for i, grid in enumerate(grids):
        for lst in (alone, together):
            r = ImogenRun(precision="mixed", **_settings(grid, "fade", False))
            r.set_state(*smooth_state(grid, seed=i, mhd=False))
            lst.append(r)
    b = ImogenBatch(together)
    b.run(9)
    for x, y in zip(alone, together):
        x.run(9)
        sx, sy = x.state(), y.state()
        assert all((sx[k] == sy[k]).all() for k in sx)
        assert x.time.time == y.time.time
    b.close()
    for r in alone + together:
        r.close()


def test_run_in_groups_stops_where_single_iterations_do():
    """img_run enqueues iterations in groups: at TIMEMAX and ITERMAX it ends in the state, time and iteration
    that one iteration at a time ends in, and can go on from there."""
    grid = (32, 32, 1)
    st = smooth_state(grid, seed=2, mhd=True)
    for lim in (dict(time_max=0.11), dict(iter_max=37), dict(time_max=1e-6)):
        s = dict(_settings(grid, "circ", True), **lim)
        a, b = ImogenRun(precision="fp64", **s), ImogenRun(precision="fp64", **s)
        for r in (a, b):
            r.set_state(*st)
        n = a.run()
        m = 0
        while b.time.running:
            m += b.run(1)
        assert n == m > 0
        assert a.time.iteration == b.time.iteration and a.time.time == b.time.time and a.progress() == b.progress()
        sa, sb = a.state(), b.state()
        assert all((sa[k] == sb[k]).all() for k in sa)
        assert a.run() == 0
        a.close()
        b.close()


PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>
#include "common.cuh"
__global__ void probe(const double* x, double* r, double* rd, double* s, double* sd, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    r[i] = img::recip(x[i]); rd[i] = 1.0 / x[i];
    s[i] = img::sqrt_goldschmidt(fabs(x[i])); sd[i] = sqrt(fabs(x[i]));
}
static double off(double a, double b) {   // in units of the last place of b; 0 for equal specials
    if (std::isnan(b)) return std::isnan(a) ? 0 : 1e9;
    if (a == b) return 0;
    if (!std::isfinite(a) || !std::isfinite(b)) return 1e9;
    return std::fabs(a - b) / (std::nextafter(std::fabs(b), INFINITY) - std::fabs(b));
}
int main() {
    std::vector<double> x = {0.0, -0.0, INFINITY, -INFINITY, NAN, 5e-324, -2.2250738585072014e-308, 1.7976931348623157e308, 1.0, -1.0};
    unsigned long long z = 88172645463325252ull;
    for (int i = 0; i < 1 << 20; ++i) {   // any bit pattern, and mantissas at ordinary exponents
        z ^= z << 13; z ^= z >> 7; z ^= z << 17;
        double v;
        unsigned long long b = i & 1 ? z : (z & 0x800fffffffffffffull) | ((unsigned long long)(1023 - 20 + z % 41) << 52);
        std::memcpy(&v, &b, 8);
        x.push_back(v);
    }
    const int n = (int)x.size();
    double *d, *o;
    cudaMalloc(&d, n * 8);
    cudaMalloc(&o, 4 * (size_t)n * 8);
    cudaMemcpy(d, x.data(), n * 8, cudaMemcpyHostToDevice);
    probe<<<(n + 255) / 256, 256>>>(d, o, o + n, o + 2 * (size_t)n, o + 3 * (size_t)n, n);
    std::vector<double> h(4 * (size_t)n);
    if (cudaMemcpy(h.data(), o, h.size() * 8, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    double wr = 0, ws = 0;
    for (int i = 0; i < n; ++i) {
        wr = std::fmax(wr, off(h[i], h[n + i]));
        ws = std::fmax(ws, off(h[2 * (size_t)n + i], h[3 * (size_t)n + i]));
    }
    std::printf("recip %g ulp, sqrt %g ulp\n", wr, ws);
    return !(wr <= 1.0 && ws <= 1.0);
}
"""


def test_reciprocal_and_square_root_within_one_ulp(tmp_path):
    """recip and sqrt_goldschmidt against the device's own division and square root: at most 1 ulp apart over
    random mantissas and bit patterns, and the same for zeros, infinities, subnormals and NaN."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    src = tmp_path / "probe.cu"
    src.write_text(PROGRAM)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17", "-I",
                    os.path.join(ROOT, "imogen_b200", "csrc"), str(src), "-o", str(tmp_path / "probe")], check=True, capture_output=True)
    r = subprocess.run([str(tmp_path / "probe")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
