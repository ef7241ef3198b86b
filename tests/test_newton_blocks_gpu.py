"""Unordered-pair kernel (lj_newton.cu) where a warp's task goes on from one
block of 256 particles to the next: every lane passes its next i's through
shared memory there while its neighbours still clear or read their sums, so
each may touch its own bytes only.

The last particles of a box are in the shortest blocks, several to a task.
Their forces after one step of a negligible dt (positions move by less than
1e-8 sigma) are held against the FP64 oracle at the MIXED force gate, 1e-5 of
max(|F|, rms F), and 10% of it for that motion; the same step from the same
state gives the same bits each time."""
import numpy as np
import pytest

import lj_testutil as U

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8193, 16384, 60001])
def test_tasks_over_several_blocks(ljgb_mod, oracle_mod, n):
    pos, vel, L = U.lattice_state(n, 0.8, 1.0, "fcc", 0.04, seed=n)
    s = ljgb_mod.System(n=n, density=0.8, temperature=1.0)
    first = None
    for _ in range(8):
        s.set_state(pos, vel)
        s.calculate_forces()
        s.integrate(1e-9)
        p, v, f = s.get_state()
        e, w = s.pair_sums()
        got = (p, v, f, e, w)
        first = first or got
        assert all(np.array_equal(a, b) for a, b in zip(got, first))
    s.close()
    r = oracle_mod.f64_forces(pos, L, True, rows=(n - 2048, n))
    assert U.force_errors(first[2][n - 2048:], r["F"])["gate_max"] <= 1.1e-5
