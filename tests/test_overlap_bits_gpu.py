"""Launches that overlap the one before them read what it wrote, not what was
there: passes that are repeated, or cut at other checkpoints, give the same bits."""
import numpy as np
import pytest

import lj_testutil as U

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [97, 700, 1500])
def test_adjoint_by_checkpoints(ljgb_mod, n):
    """The backward pass replays a segment of the forward pass from its
    checkpoint: whatever the segments are, the states and gradients agree."""
    pos, vel, _ = U.lattice_state(n, 0.8, 1.0, "fcc", 0.04, seed=n)
    out = []
    for every in (1, 3, 12, 12):
        a = ljgb_mod.Adjoint(n=n, density=0.8, temperature=1.0, checkpoint_every=every)
        a.set_state(pos, vel)
        for _ in range(3):
            loss = a.forward(0.004, 12)
            g = a.backward()
            out.append((np.float64(loss),) + tuple(np.asarray(x) for x in g))
        a.close()
    for got in out[1:]:
        assert all(np.array_equal(x, y) for x, y in zip(got, out[0]))


@pytest.mark.parametrize("n", [300, 4000])
def test_uploads_in_turn(ljgb_mod, n):
    """Two states uploaded in turn: each step starts from the one just given."""
    sets = [U.lattice_state(n, 0.7, 1.0, "fcc", 0.05, seed=k)[:2] for k in (1, 2)]
    s = ljgb_mod.System(n=n, density=0.7, temperature=1.0)
    first = {}
    for turn in range(40):
        s.set_state(*sets[turn % 2])
        s.calculate_forces()
        s.integrate(0.004)
        got = s.get_state()
        want = first.setdefault(turn % 2, got)
        assert all(np.array_equal(x, y) for x, y in zip(got, want)), turn
    s.close()
