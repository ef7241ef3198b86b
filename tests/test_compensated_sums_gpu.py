"""Sums of the MIXED step keep what meets a much larger term elsewhere.

One particle has two neighbours on opposite sides, so near that each pushes with
1e9, exactly cancelling (their fixed-point separations are negatives of each
other), and a third that pulls with 1.2 along the same line; all others are 15
sigma or more away (1.4e-7 each at most).  The three are placed so that no two
are in one plain FP32 sum of 32 pairs of the step's kernel and all are in one of
its TwoSum sums: the third's pull then comes through whole, and the force is held
to the MIXED gate, 1e-5 of it (an uncompensated addition of 1.2 to 1e9 keeps
multiples of 64).  The time step is so small that no position changes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NEAR, PULL = 0.274, 1.5


def _force(d):
    r2 = (d * d).sum(-1, keepdims=True)
    i6 = r2 ** -3
    return 24.0 * i6 * (2.0 * i6 - 1.0) / r2 * d


def _check(ljgb, n, L, centre, push, push_back, pull):
    s = ljgb.System(n=n, density=n / L ** 3, temperature=1.0)
    L = s.L
    unit = 3 * L / 2 ** 32                       # the shadow's grid, as whole numbers below
    m = np.arange(0.5, L, 4.0)
    sites = np.stack(np.meshgrid(m, m, m, indexing="ij"), -1).reshape(-1, 3)
    mid = np.full(3, np.floor(L / 2 / unit))
    d = sites - mid * unit
    d -= L * np.round(d / L)
    order = np.argsort(-(d * d).sum(1), kind="stable")[:n - 4]
    assert (d[order] ** 2).sum(1).min() > 15.0 ** 2
    grid = np.empty((n, 3))
    grid[[centre, push, push_back, pull]] = mid + np.array([[0, 0, 0], [NEAR, 0, 0], [-NEAR, 0, 0], [PULL, 0, 0]]) / unit
    grid[[i for i in range(n) if i not in (centre, push, push_back, pull)]] = sites[order] / unit
    grid = np.round(grid)
    grid[push_back] = 2 * grid[centre] - grid[push]
    s.set_state(grid * unit, np.zeros((n, 3)))
    s.calculate_forces()
    s.integrate(1e-10)
    got = s.get_state()[2][centre]
    s.close()
    d = grid[centre] - np.delete(grid, [centre], 0)
    want = _force((d - 2 ** 32 / 3 * np.round(d / (2 ** 32 / 3))) * unit)
    big = np.abs(want).max()
    want = want.sum(0)
    assert 5e8 < big < 5e9 and 1.0 < abs(want[0]) < 1.3, (big, want)
    assert np.abs(got - want).max() <= 1e-5 * abs(want[0]), (got, want)


@pytest.mark.parametrize("n", [700, 2000])
def test_row_step(ljgb_mod, n):
    """Lanes 1, 2 and 3 of a warp's j's."""
    _check(ljgb_mod, n, 60.0, 0, 33, 66, 99)


@pytest.mark.parametrize("n", [256, 400, 512])
def test_cluster_step(ljgb_mod, n):
    """Lanes 1, 2 and 3 of a group of eight, in a warp's part of the j's."""
    _check(ljgb_mod, n, 60.0, 0, 9, 18, 27)


def test_unordered_pair_step(ljgb_mod):
    """A j of the second block's first tile and i's of the first block: the push
    and the pull in the two halves of the same eight turns, the push back in
    another eight."""
    _check(ljgb_mod, 8192, 100.0, 261, 5, 27, 36)
