"""Pair histogram at the edges of its blocks (256 i's) and chunks (32 j's)."""
import numpy as np
import pytest

import lj_testutil as U

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [2, 31, 33, 255, 256, 257, 288, 513, 5000])
@pytest.mark.parametrize("boundary", [0, 1])
def test_rdf_counts_at_block_edges(ljgb_mod, oracle_mod, N, boundary):
    """Every mode against the exact emulation: each unordered pair is
    evaluated once and counted twice, whatever the ragged ends.  A walled
    box's shadow comes from its own frame, so there only the totals are known
    exactly (every ordered pair in the clamped mode)."""
    rho = 0.4
    pos, vel, L = U.lattice_state(N, rho, 1.0, "fcc", 0.05, seed=N)
    s = ljgb_mod.System(n=N, density=rho, boundary=boundary)
    s.set_state(pos, vel)
    dr = L / 2 / 100
    clamp, drop, lin = s.rdf_counts(0, 64, 0.3), s.rdf_counts(1, 64, 0.3), s.rdf_counts(2, 100, dr)
    assert clamp.sum() == N * (N - 1)
    assert np.array_equal(clamp[:63], drop[:63]) and (drop % 2 == 0).all() and (lin % 2 == 0).all()
    if boundary == 0:
        q = oracle_mod.emu_fixed(pos, L)
        ks = L / 4294967296.0
        k2 = np.float32(ks * ks)
        assert np.array_equal(clamp, oracle_mod.emu_rdf_r2(q, k2, np.float32(1.0 / 0.3), 64, 0))
        assert np.array_equal(drop, oracle_mod.emu_rdf_r2(q, k2, np.float32(1.0 / 0.3), 64, 1))
        rmax = 100 * dr
        assert np.array_equal(lin, oracle_mod.emu_rdf_r(q, k2, np.float32(1.0 / dr), np.float32(rmax * rmax), 100))
    s.close()
