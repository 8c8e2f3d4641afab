"""Batches of grids of many sizes share launches (GPU required): members whose CTAs pad to the same block size go into
one launch, with idle threads, and equal their runs alone bit for bit."""
import numpy as np
import pytest

from imogen_b200 import ImogenBatch, ImogenRun
from tests.parity import smooth_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("bc,magnet,dims", [("circ", False, 2), ("circ", True, 2), ("fade", False, 2), ("const", True, 3), ("fade", False, 3)])
def test_grids_of_many_sizes_share_launches(bc, magnet, dims, precision):
    rng = np.random.default_rng(2)
    sides = np.exp(rng.uniform(np.log(24), np.log(150 if dims == 2 else 40), 24)).astype(int)
    runs, alone = [], []
    for i, n in enumerate(sides):
        grid = (int(n), int(n) + i % 3, 1 if dims == 2 else int(n))
        for lst in (runs, alone):
            r = ImogenRun(precision=precision, grid=grid, dgrid=(1 / 64,) * 3, gamma=5 / 3, cfl=0.35, bc=bc, limiter="vanleer",
                          magnet=magnet, time_max=1e5, iter_max=10 ** 6)
            r.set_state(*smooth_state(grid, seed=i, mhd=magnet))
            lst.append(r)
    b = ImogenBatch(runs)
    b.run(14)
    before = b.launches
    b.run(6)
    launches = (b.launches - before) / 6
    for x, y in zip(runs, alone):
        y.run(20)
        sx, sy = x.state(), y.state()
        assert all((sx[k] == sy[k]).all() for k in sx), x.grid
    # two timesteps of `dims` fluid sweeps and twice as many magnet kernels, at most 8 block sizes each (FP32
    # also two forms of the fluxes), 2 time updates and their passes
    assert launches <= 2 * dims * 8 * (3 if magnet else 1) + 4, launches
    b.close()
    for r in runs + alone:
        r.close()


def test_members_on_the_tile_kernels_equal_their_runs_alone(monkeypatch):
    """Contexts created with IMOGEN_B200_TILE_KERNELS=1 keep the tile kernels in a batch that fills the chip."""
    monkeypatch.setenv("IMOGEN_B200_TILE_KERNELS", "1")
    runs, alone = [], []
    for i, n in enumerate((200, 150, 260, 90, 230)):
        for lst in (runs, alone):
            r = ImogenRun(precision="mixed", grid=(n, n + i, 1), dgrid=(1 / 64,) * 3, gamma=5 / 3, cfl=0.35, bc="circ", limiter="vanleer",
                          magnet=True, time_max=1e5, iter_max=10 ** 6)
            assert not any(t[6] for t in r.tiling("fluid").values())
            r.set_state(*smooth_state((n, n + i, 1), seed=i, mhd=True))
            lst.append(r)
    b = ImogenBatch(runs)
    b.run(9)
    for x, y in zip(runs, alone):
        y.run(9)
        sx, sy = x.state(), y.state()
        assert all((sx[k] == sy[k]).all() for k in sx), x.grid
    b.close()
    for r in runs + alone:
        r.close()
