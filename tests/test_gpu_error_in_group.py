"""img_run enqueues iterations in groups: an error inside one leaves the state, the time and the iteration that one
iteration at a time leaves (GPU required; long x pencils, whose launches over a thread-block cluster cannot look at
an error that is raised while they run)."""
import numpy as np
import pytest

from imogen_b200 import ImogenError, ImogenRun

pytestmark = pytest.mark.gpu

GRID = (4099, 3, 3)
SEGMENT = (1, 1025, 3, 352, 4, 1, 1)      # over a cluster of 3


def _state(overflow):
    """A gas at rest with one slightly warmer cell per pencil, above the 1e-2 speed floor until it has spread (a CFL
    error after some iterations), or with an energy whose flux differences overflow in the first."""
    rho = np.ones(GRID)
    mom, mag = np.zeros((3,) + GRID), np.zeros((3,) + GRID)
    P = np.full(GRID, 4e-5)
    if overflow:
        mom[0] = 0.1 * np.sin(np.arange(GRID[0]))[:, None, None]
        P[:] = 1.0
        P[2000] = 3e38 if overflow == "mixed" else 1e308
    else:
        P[2000] = 9e-5
    return rho, mom, P / (2 / 3), mag


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("tile", [False, True])
@pytest.mark.parametrize("overflow", [False, True])
def test_error_inside_a_group_leaves_what_single_iterations_leave(overflow, tile, precision, monkeypatch):
    s = dict(grid=GRID, dgrid=(1 / 4096,) * 3, gamma=5 / 3, cfl=0.35, bc={"x": "const", "y": "circ", "z": "circ"}, magnet=False,
             time_max=1e5, iter_max=10 ** 6)
    st = _state(overflow and precision)
    monkeypatch.setenv("IMOGEN_B200_TILE_KERNELS", "1" if tile else "0")
    ends = []
    for one_by_one in (True, False):
        r = ImogenRun(precision=precision, **s)
        if not tile:
            r.set_tiling(1, SEGMENT)
        t = r.tiling("fluid")[1]
        assert t[2] > 1 and bool(t[6]) != tile
        r.set_state(*st)
        with pytest.raises(ImogenError) as e:
            if one_by_one:
                for _ in range(200):
                    r.run(1)
            r.run(200)
        got = [r.download(k) for k in ("mass", "momx", "momy", "momz", "ener")]
        r.time.set(0.0, 0.0, 1)          # clears the error
        ends.append((e.value.code, got))
        r.close()
    (ca, a), (cb, b) = ends
    assert ca == cb
    assert all(np.array_equal(x, y, equal_nan=True) for x, y in zip(a, b))
