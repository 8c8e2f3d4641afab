"""Segment fluid and window magnet kernels on long pencils (GPU required): two pencils per CTA along y, periodic pencils
along x over a thread-block cluster whose last segment has one, two or three cells, and batches whose members round the
FP32 fluxes in different forms.  Against the C++ oracle, relative L1 at most 1e-11 (FP64) and 2e-5 (mixed) after 4
iterations, as in test_gpu_segment_edges.py; a batch equals its members alone bit for bit."""
import pytest

from imogen_b200 import ImogenBatch, ImogenRun
from tests.parity import errors, make_pair, smooth_state

pytestmark = pytest.mark.gpu
TOL = {"fp64": 1e-11, "mixed": 2e-5}


def _settings(grid, bc, magnet=True, limiter=("vanleer", "minmod", "superbee")):
    return dict(grid=grid, dgrid=(1.0 / max(grid),) * 3, gamma=5 / 3, cfl=0.35, bc=bc, limiter=limiter, magnet=magnet, time_max=1e5,
                iter_max=10 ** 6)


def _check(s, precision, tilings=()):
    o, g = make_pair(s, smooth_state(s["grid"], seed=9, mhd=True), precision=precision)
    for kind, dim, t in tilings:
        g.set_tiling(dim, t, kind=kind)
        assert g.tiling(kind)[dim] == t
    o.run(4)
    g.run(4)
    e = errors(g.state(), o.state())
    t = g.tiling("fluid")
    g.close()
    assert all(v <= TOL[precision] for v in e.values()), e
    return t


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("bc", ["circ", "const"])
@pytest.mark.parametrize("grid", [(16, 1021, 1), (24, 700, 1), (17, 6, 601)])
def test_two_pencils_per_block_across(grid, bc, precision):
    d = 2 if grid[2] == 1 else 3
    t = _check(_settings(grid, bc), precision)[d]
    if precision == "mixed" or grid[d - 1] < 850:   # (two longer FP64 pencils do not fit: the tile kernels)
        assert t[0] == 2 and t[6] == 1, t


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [4801, 4802, 4803])
@pytest.mark.parametrize("cells,cl", [(4, 3), (4, 5), (8, 3)])
def test_periodic_pencils_over_a_cluster_with_a_short_last_segment(cells, cl, n, precision):
    s = -(-n // cells)
    t = (1, s, cl, -(-(-(-s // cl)) // 32) * 32, cells, 1, 1)
    tilings = [("magnet", 1, t)] + ([("fluid", 1, t)] if precision == "mixed" or cells < 8 else [])
    _check(_settings((n, 3, 3), "circ"), precision, tilings)


def test_members_of_different_flux_forms_in_a_batch_equal_their_runs_alone():
    grids = [(64, 48, 1), (75, 33, 1), (52, 90, 1), (128, 64, 1), (61, 47, 1), (96, 100, 1)]
    alone, together = [], []
    for i, grid in enumerate(grids):
        for lst in (alone, together):
            r = ImogenRun(precision="mixed", **_settings(grid, "circ", limiter="vanleer"))
            r.set_state(*smooth_state(grid, seed=i, mhd=True))
            lst.append(r)
    b = ImogenBatch(together)
    b.run(9)
    for x, y in zip(alone, together):
        x.run(9)
        sx, sy = x.state(), y.state()
        assert all((sx[k] == sy[k]).all() for k in sx)
    b.close()
    for r in alone + together:
        r.close()
