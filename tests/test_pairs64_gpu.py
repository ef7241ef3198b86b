"""FP64 pair pass over unordered pairs, at the edges of its tiles (32
particles), task splits (8, 4, 2, 1 tasks a square) and square sides, against
the FP64 oracle.  Both sum the same terms in different orders: the 1e-11 of
the FP64 gate is far above what ordering can do (N^1/2 2^-53 relative to the
largest term) and far below any missing or doubled pair."""
import numpy as np
import pytest

import lj_testutil as U

pytestmark = pytest.mark.gpu

TOL = 1e-11


def _check(oracle_mod, s, pos, L, periodic, sigma, rows=None):
    r = oracle_mod.f64_forces(pos, L, periodic, 1.0, sigma, rows=rows)
    _, _, F = s.get_state()
    e, w = s.pair_sums()
    i0, i1 = (0, s.n) if rows is None else rows
    assert U.force_errors(F[i0:i1], r["F"])["gate_max"] <= TOL
    assert np.abs(e[i0:i1] - r["e"]).max() <= TOL * np.abs(r["e"]).max()
    if rows is None:
        o = s.observables()
        assert o["V"] == pytest.approx(r["V"], rel=TOL, abs=1e-9)
        assert o["W"] == pytest.approx(r["W"], rel=TOL, abs=1e-9)
    # every pair's two forces are exact negatives: the sums cancel to rounding
    assert np.abs(F.sum(0)).max() <= 1e-12 * np.abs(F).sum()


@pytest.mark.parametrize("boundary,sigma", [(0, 1.0), (0, 1.1), (1, 1.0), (2, 0.9)])
@pytest.mark.parametrize("N", [2, 31, 32, 33, 64, 65, 500, 513, 1000, 1601, 2500])
def test_tile_edges(ljgb_mod, oracle_mod, N, boundary, sigma):
    pos, vel, L = U.lattice_state(N, 0.4, 1.0, "fcc", 0.05, seed=N)
    s = ljgb_mod.System(n=N, density=0.4, boundary=boundary, precision=1, sigma=sigma)
    s.set_state(pos, vel)
    s.calculate_forces()
    _check(oracle_mod, s, pos, L, boundary == 0, sigma)
    s.close()


def test_squares_of_several_tiles(ljgb_mod, oracle_mod):
    """N = 10001: squares of two tiles, j sums carried from row to row."""
    N = 10001
    pos, vel, L = U.lattice_state(N, 0.85, 1.0, "fcc", 0.05, seed=3)
    s = ljgb_mod.System(n=N, density=0.85, precision=1)
    s.set_state(pos, vel)
    s.calculate_forces()
    for rows in ((0, 96), (4990, 5060), (N - 70, N)):
        _check(oracle_mod, s, pos, L, True, 1.0, rows=rows)
    s.close()


def test_particles_outside_the_box(ljgb_mod, oracle_mod):
    """Separations of several periods take the image of the nearest one."""
    N = 300
    pos, vel, L = U.lattice_state(N, 0.4, 1.0, "fcc", 0.05, seed=8)
    moved = pos + L * np.random.default_rng(2).integers(-3, 4, pos.shape)
    a = ljgb_mod.System(n=N, density=0.4, precision=1)
    a.set_state(moved, vel)
    a.calculate_forces()
    r = oracle_mod.f64_forces(moved, L, True, 1.0, 1.0)
    assert U.force_errors(a.get_state()[2], r["F"])["gate_max"] <= TOL
    a.close()


def test_uneven_fp64_batch(ljgb_mod, oracle_mod):
    sizes = [33, 700, 32, 250]
    cfgs = [ljgb_mod.config(n=n, density=0.3 + 0.1 * k, precision=1, boundary=k % 3, lattice=1, jitter=0.05, seed=k + 1)
            for k, n in enumerate(sizes)]
    b = ljgb_mod.System(batch=cfgs)
    pos, _, F = b.get_state()
    for k, c in enumerate(cfgs):
        sl = slice(b.offsets[k], b.offsets[k + 1])
        L = (c.n / c.density) ** (1 / 3)
        r = oracle_mod.f64_forces(pos[sl], L, c.boundary == 0, 1.0, 1.0)
        assert U.force_errors(F[sl], r["F"])["gate_max"] <= TOL, k
    b.close()
