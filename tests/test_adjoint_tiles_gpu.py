"""The adjoint's pair passes at the edges of their tiles (32 particles) and of
the splits of a square (4 tasks: N = 33, 100; 2: 300, 1000; 1: 500; one warp a
task: 1601), against the numpy adjoint with the tolerances of
test_adjoint.py: FP64 sums of the same terms in another order."""
import numpy as np
import pytest

import lj_testutil as U

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [33, 100, 300, 500, 1000, 1601])
def test_adjoint_at_tile_edges(ljgb_mod, N):
    import adjoint as A
    rho, dt, S, wts = 0.6, 0.004, 3, (0.3, 0.7, 0.2)
    pos, vel, _ = U.lattice_state(N, rho, 1.0, "fcc", 0.02, seed=N)
    t = A.Trajectory(pos, vel, rho, 1.1, 0.95, wts)
    loss_ref = t.forward(dt, S)
    de_r, ds_r, dx_r, dv_r = t.backward()
    adj = ljgb_mod.Adjoint(n=N, density=rho, temperature=1.0, epsilon=1.1, sigma=0.95, checkpoint_every=2)
    adj.set_state(pos, vel)
    adj.set_loss(*wts)
    assert adj.forward(dt, S) == pytest.approx(loss_ref, rel=1e-11)
    de, ds, dx, dv = adj.backward()
    assert de == pytest.approx(de_r, rel=1e-9)
    assert ds == pytest.approx(ds_r, rel=1e-9)
    assert np.abs(dx - dx_r).max() <= 1e-9 * np.abs(dx_r).max()
    assert np.abs(dv - dv_r).max() <= 1e-9 * np.abs(dv_r).max()
