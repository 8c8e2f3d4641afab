"""Tilings that img_set_tiling has long accepted (GPU required): short pencils held whole by one thread in the largest
CTAs, 32 FP64 pencils side by side, hundreds of short pencils along x in one CTA of the window kernels, and, with fade
ends, segment tilings whose CTA has no room for the anchors of the ends, which leave the sweep to the tile kernels.
Results against the C++ oracle, relative L1 at most 1e-11 (FP64) and 2e-5 (mixed) after 4 iterations, as in
test_gpu_segment_edges.py."""
import pytest

from tests.parity import errors, make_pair, smooth_state

pytestmark = pytest.mark.gpu
TOL = {"fp64": 1e-11, "mixed": 2e-5}

CASES = [
    ("fluid", (512, 3, 3), "circ", 2, (512, 1, 1, 512, 3, 1, 1), ("mixed",)),
    ("fluid", (512, 3, 3), "circ", 3, (256, 1, 1, 256, 3, 1, 1), ("mixed", "fp64")),
    ("fluid", (128, 4, 4), "const", 2, (512, 1, 1, 512, 4, 1, 1), ("mixed",)),
    ("fluid", (26, 26, 26), "const", 2, (32, 13, 1, 416, 2, 1, 1), ("fp64",)),
    ("fluid", (52, 39, 26), "circ", 3, (32, 13, 1, 416, 2, 1, 1), ("fp64",)),
    ("fluid", (26, 26, 26), "fade", 3, (32, 13, 1, 416, 2, 1, 1), ("fp64",)),
    ("magnet", (6, 100, 100), "circ", 1, (256, 2, 1, 512, 4, 1, 1), ("mixed", "fp64")),
    ("magnet", (5, 400, 1), "const", 1, (128, 3, 1, 384, 2, 1, 1), ("mixed", "fp64")),
    ("magnet", (3, 60, 60), "circ", 1, (512, 1, 1, 512, 8, 1, 1), ("mixed",)),
]


@pytest.mark.parametrize("kind,grid,bc,dim,tiling,precision", [(*c[:5], p) for c in CASES for p in c[5]])
def test_tiling_is_accepted_and_runs(kind, grid, bc, dim, tiling, precision):
    s = dict(grid=grid, dgrid=(1.0 / max(grid),) * 3, gamma=5 / 3, cfl=0.35, bc=bc, limiter="vanleer", magnet=kind == "magnet",
             time_max=1e5, iter_max=10 ** 6)
    o, g = make_pair(s, smooth_state(grid, seed=6, mhd=kind == "magnet"), precision=precision)
    g.set_tiling(dim, tiling, kind=kind)
    assert g.tiling(kind)[dim] == tiling
    o.run(4)
    g.run(4)
    e = errors(g.state(), o.state())
    g.close()
    assert all(v <= TOL[precision] for v in e.values()), e
