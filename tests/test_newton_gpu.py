"""Unordered-pair step (lj_newton.cu) at the edges of its tiles (32) and
blocks (256), against the FP64 path with the tolerances of
tests/test_rows_gpu.py."""
import numpy as np
import pytest

import lj_testutil as U

pytestmark = pytest.mark.gpu

DT, STEPS = 0.004, 4


@pytest.mark.parametrize("canonical", [0, 1])
@pytest.mark.parametrize("N,boundary", [(8191, 0), (8192, 0), (8192, 1), (8193, 0), (8223, 1), (8225, 0), (8447, 0),
                                        (8449, 1), (16384, 0), (20011, 0)])
def test_newton_step_matches_fp64(ljgb_mod, N, boundary, canonical):
    pos, vel, L = U.lattice_state(N, 0.7, 1.1, "fcc", 0.05, seed=N)
    out = []
    for prec in (0, 1):
        s = ljgb_mod.System(n=N, density=0.7, temperature=1.1, canonical=canonical, boundary=boundary, precision=prec)
        s.set_state(pos, vel)
        s.calculate_forces()
        s.integrate(DT, STEPS - 1)
        s.integrate(DT)
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


def test_newton_step_by_route(ljgb_mod):
    """Records and observables do not depend on how the steps are divided, on
    the graphs' route, or on the autotuner's choice beyond rounding."""
    kw = dict(n=8500, density=0.8, temperature=1.0, canonical=1, lattice=ljgb_mod.LATTICE_FCC, jitter=0.03, seed=6)
    runs = []
    for route in range(3):
        s = ljgb_mod.System(**kw)
        s.set_recording(16)
        if route == 2:
            s.counters_configure([(0, 10, 0.1, 0.0)])
        for part in (5, 1, 2):
            s.integrate(DT, part)
            if route == 1:
                s.observables()
        runs.append((s.records(16), s.observables(), s.get_state()))
        s.close()
    for recs, o, st in runs[1:]:
        assert recs == runs[0][0] and len(recs) == 8
        assert o == runs[0][1]
        assert all(np.array_equal(a, b) for a, b in zip(st, runs[0][2]))
    s = ljgb_mod.System(**kw)
    s.autotune()
    s.integrate(DT, 8)
    for k in ("U", "K", "P", "t", "step"):
        assert s.observables()[k] == pytest.approx(runs[0][1][k], rel=1e-6), k
    s.close()


def test_newton_launches(ljgb_mod):
    for canonical, per_step in ((1, 3), (0, 2)):
        s = ljgb_mod.System(n=9000, density=0.8, temperature=1.0, canonical=canonical)
        c0 = s.launch_count()
        s.integrate(DT, 4)
        assert s.launch_count() - c0 == 1 + per_step * 4      # predictor; pairs, sums (, close)
        s.close()
