"""The FP32 rounding of the segment fluid kernels (GPU required).  The flows these grids carry grow a difference in the
last bit by several powers of ten in a hundred iterations, so a kernel that replaces another on the same grid has to
round as it did: one sweep of the segment kernels equals one of the pencil-tile kernels (IMOGEN_B200_TILE_KERNELS=1)
bit for bit."""
import numpy as np
import pytest

from imogen_b200 import ImogenRun

pytestmark = pytest.mark.gpu
F32 = lambda a: np.asarray(a, dtype=np.float32).astype(np.float64)


def _settings(grid, bc, magnet):
    return dict(grid=grid, dgrid=(1 / 256,) * 3, gamma=5 / 3, cfl=0.35, bc=bc, limiter="vanleer", magnet=magnet,
                time_max=1e5, iter_max=10 ** 6)


def _sweep(settings, state, X, dt, tile, monkeypatch):
    """One fluid sweep along X, not a run's first (the first capture takes the tile kernels on either side)."""
    monkeypatch.setenv("IMOGEN_B200_TILE_KERNELS", "1" if tile else "0")
    r = ImogenRun(precision="mixed", **settings)
    assert bool(r.tiling("fluid")[X][6]) != tile
    r.set_state(*state(r))
    r.time.set(0.0, 0.0, 1)
    r.relaxing_fluid(2 if X == 1 else 1)   # with dt = 0: changes nothing
    r.time.set(0.0, dt, 1)
    r.relaxing_fluid(X)
    out = [r.download(k).astype(np.float32) for k in ("mass", "momx", "momy", "momz", "ener")]
    r.close()
    return out


def _pressure_residue(grid, X, seed):
    """A state at rest along X whose 'totsnd' pressure is what the FP32 rounding of E leaves of terms 1e7 times
    larger.  With a tiny dt the new momentum along X shows the FP32 pressure alone, and an FP64 sum rounded in another
    order shows in a few cells of a hundred."""
    def state(run):
        rng = np.random.default_rng(seed)
        rho, mom, mag = F32(rng.uniform(0.5, 2, grid)), F32(rng.uniform(-1, 1, (3,) + grid)), F32(rng.uniform(-1, 1, (3,) + grid))
        mom[X - 1] = mag[X - 1] = 0
        run.set_state(rho, mom, rho, mag)   # for the cell-centred field
        msq = sum(run.download(k) ** 2 for k in ("cmagx", "cmagy", "cmagz"))
        at = 0.5 * (mom ** 2).sum(0) / rho - msq / 4   # (gamma - 1) (E - kinetic) + (2 - gamma) B^2 / 2 = 0
        ener = F32(at)
        return rho, mom, np.where(ener < at, F32(np.nextafter(ener.astype(np.float32), np.float32(9))), ener), mag
    return state


@pytest.mark.parametrize("bc", ["circ", "const"])
@pytest.mark.parametrize("grid,X", [((64, 64, 16), 1), ((64, 64, 16), 2), ((16, 16, 64), 3), ((75, 32, 9), 1), ((32, 75, 9), 2)])
def test_pressure_rounds_as_in_the_tile_kernels(grid, X, bc, monkeypatch):
    s = _settings(grid, bc, True)
    a, b = (_sweep(s, _pressure_residue(grid, X, 7), X, 1e-20, tile, monkeypatch) for tile in (False, True))
    assert np.count_nonzero(a[X]) > 0.9 * a[X].size
    assert all((x == y).all() for x, y in zip(a, b)), [int((x != y).sum()) for x, y in zip(a, b)]


def _ordinary(grid, magnet, seed):
    def state(run):
        rng = np.random.default_rng(seed)
        rho, mom = rng.uniform(0.5, 2, grid), rng.uniform(-1, 1, (3,) + grid)
        mag = rng.uniform(-1, 1, (3,) + grid) if magnet else np.zeros((3,) + grid)
        return rho, mom, 1 + 0.5 * (mom ** 2).sum(0) / rho + 0.5 * (mag ** 2).sum(0), mag
    return state


@pytest.mark.parametrize("magnet", [False, True])
@pytest.mark.parametrize("grid,bc,X", [((48, 40, 1), "fade", 1), ((48, 41, 1), "fade", 2), ((24, 22, 67), "fade", 3), ((500, 24, 1), "fade", 1),
                                       ((61, 40, 1), {"x": ("fade", "const"), "y": "fade", "z": "circ"}, 1),
                                       ((40, 61, 1), {"x": "fade", "y": ("circ", "fade"), "z": "circ"}, 2)])
def test_fade_ends_round_as_in_the_tile_kernels(grid, bc, X, magnet, monkeypatch):
    s = _settings(grid, bc, magnet)
    a, b = (_sweep(s, _ordinary(grid, magnet, 5), X, 1e-3, tile, monkeypatch) for tile in (False, True))
    assert all((x == y).all() for x, y in zip(a, b)), [int((x != y).sum()) for x, y in zip(a, b)]


def _tilings(n, d, precision="mixed"):
    """Segment tilings of a pencil of n cells along dimension d, one CTA of at least 64 threads, for each number of cells
    a thread that may hold (of 3-cell pencils, 3)."""
    out = []
    for c in (2, 3, 4, 8):
        if c == 3 and n % 3 or n == 3 and c != 3:
            continue
        s = -(-n // c)
        for wb in (1, 2, 4, 8, 16, 32) if d == 1 else (4, 8, 16, 32):
            nt = -(-wb * s // 32) * 32
            if 64 <= nt <= 512:
                out.append((wb, s, 1, nt, c, 1, 1))
                break
    return out


FORMS = [((384, 24, 1), 1), ((24, 48, 1), 2), ((75, 24, 1), 1), ((24, 90, 1), 2), ((24, 24, 51), 3)]


def _tiled_sweep(grid, X, magnet, tiling=None):
    r = ImogenRun(precision="mixed", **_settings(grid, "circ", magnet))
    r.set_state(*_ordinary(grid, magnet, 3)(None))
    if tiling:
        r.set_tiling(X, tiling)
    used = r.tiling("fluid")[X]
    r.time.set(0.0, 0.0, 1)
    r.relaxing_fluid(2 if X == 1 else 1)
    r.time.set(0.0, 1e-3, 1)
    r.relaxing_fluid(X)
    out = [r.download(k) for k in ("mass", "momx", "momy", "momz", "ener")]
    r.close()
    return used, out


@pytest.mark.parametrize("magnet", [False, True])
@pytest.mark.parametrize("grid,X", FORMS)
def test_any_picked_segment_tiling_rounds_alike(grid, X, magnet):
    """The default tiling picked and every other number of cells a thread give the same bits; so does the default
    itself on grids of whole 4-cell segments that fill CTAs (the first two)."""
    default, plain = _tiled_sweep(grid, X, magnet)
    assert default[6]
    want = _tiled_sweep(grid, X, magnet, default)[1]
    tried = _tilings(grid[X - 1], X)
    assert len({t[4] for t in tried}) >= 3
    for t in tried:
        got = _tiled_sweep(grid, X, magnet, t)[1]
        assert all((x == y).all() for x, y in zip(want, got)), t
    if grid in ((384, 24, 1), (24, 48, 1)):
        assert all((x == y).all() for x, y in zip(want, plain))
