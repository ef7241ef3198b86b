"""The row step (lj_rows.cu) on boxes that the cluster kernel takes otherwise:
with a counter configured they step one launch at a time.  Against the FP64 path
over the same steps, with the bounds of tests/test_rows_gpu.py: the MIXED gate
(forces within 1e-5 of max(|F|, rms F)) adds at most dt 1e-5 max|F| a step to a
velocity, and dt times that to a position."""
import numpy as np
import pytest

import lj_testutil as U

pytestmark = pytest.mark.gpu

DT, STEPS = 0.004, 6


@pytest.mark.parametrize("canonical", [0, 1])
@pytest.mark.parametrize("boundary", [0, 1])
@pytest.mark.parametrize("N", [2, 3, 31, 33, 64, 151, 301, 302, 303, 511, 512])
def test_row_step_matches_fp64(ljgb_mod, N, boundary, canonical):
    pos, vel, L = U.lattice_state(N, 0.6, 1.1, "fcc", 0.05, seed=N)
    out = []
    for prec in (0, 1):
        s = ljgb_mod.System(n=N, density=0.6, temperature=1.1, canonical=canonical, boundary=boundary, precision=prec)
        s.counters_configure([(0, 10, 0.1, 0.0)])
        s.set_state(pos, vel)
        s.calculate_forces()
        c0 = s.launch_count()
        s.integrate(DT, STEPS - 1)
        s.integrate(DT)
        if prec == 0:
            assert s.launch_count() - c0 >= (3 if canonical else 2) * STEPS
        out.append((s.get_state(), s.observables(), s.pair_sums()))
        s.close()
    (p0, v0, f0), o0, (e0, w0) = out[0]
    (p1, v1, f1), o1, (e1, w1) = out[1]
    assert U.force_errors(f0, f1)["gate_max"] <= 2e-5
    fmax = max(1.0, np.abs(f1).max())
    assert np.abs(v0 - v1).max() <= DT * STEPS * 1e-5 * fmax
    d = np.abs(p0 - p1)
    if boundary == 0:
        d = np.minimum(d, L - d)
    assert d.max() <= DT * DT * STEPS * STEPS * 1e-5 * fmax
    assert np.abs(e0 - e1).max() <= 2e-5 * np.abs(e1).max() and np.abs(w0 - w1).max() <= 2e-5 * np.abs(w1).max()
    for k in ("K", "V", "U", "T", "av_U_tot", "t", "Tkin_tvn"):
        assert o0[k] == pytest.approx(o1[k], rel=1e-5, abs=1e-5 * N), k
    assert o0["step"] == o1["step"] == STEPS and o0["av_iters"] == o1["av_iters"]
