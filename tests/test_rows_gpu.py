"""Row step (lj_rows.cu) at the edges of its rows, chunks (32 j's) and tiles
(2048 j's), against the FP64 path over the same steps.

Tolerance: the MIXED gate (forces within 1e-5 of max(|F|, rms F)) bounds what
one step can add to a velocity by dt 1e-5 max|F|; over the 6 steps here that
is dt * 6 * 1e-5 max|F| for velocities, and dt times that for positions."""
import numpy as np
import pytest

import lj_testutil as U

pytestmark = pytest.mark.gpu

DT, STEPS = 0.004, 6


@pytest.mark.parametrize("canonical", [0, 1])
@pytest.mark.parametrize("boundary", [0, 1])
@pytest.mark.parametrize("N", [2, 3, 31, 33, 64, 301, 302, 605, 2047, 2049, 4097, 8200, 13001])
def test_row_step_matches_fp64(ljgb_mod, N, boundary, canonical):
    pos, vel, L = U.lattice_state(N, 0.6, 1.1, "fcc", 0.05, seed=N)
    out = []
    for prec in (0, 1):
        s = ljgb_mod.System(n=N, density=0.6, temperature=1.1, canonical=canonical, boundary=boundary, precision=prec)
        s.set_state(pos, vel)
        s.calculate_forces()
        s.integrate(DT, STEPS - 1)
        s.integrate(DT)
        out.append((s.get_state(), s.observables(), s.pair_sums()))
        s.close()
    (p0, v0, f0), o0, (e0, w0) = out[0]
    (p1, v1, f1), o1, (e1, w1) = out[1]
    assert U.force_errors(f0, f1)["gate_max"] <= 2e-5   # 1e-5 of the pass, 1e-5 for the drifted positions
    fmax = max(1.0, np.abs(f1).max())
    assert np.abs(v0 - v1).max() <= DT * STEPS * 1e-5 * fmax
    d = np.abs(p0 - p1)
    if boundary == 0:
        d = np.minimum(d, L - d)                        # a wrap one step earlier or later
    assert d.max() <= DT * DT * STEPS * STEPS * 1e-5 * fmax
    assert np.abs(e0 - e1).max() <= 2e-5 * np.abs(e1).max() and np.abs(w0 - w1).max() <= 2e-5 * np.abs(w1).max()
    for k in ("K", "V", "U", "T", "av_U_tot", "t", "Tkin_tvn"):
        assert o0[k] == pytest.approx(o1[k], rel=1e-5, abs=1e-5 * N), k
    assert o0["step"] == o1["step"] == STEPS and o0["av_iters"] == o1["av_iters"]


@pytest.mark.parametrize("canonical", [0, 1])
def test_row_step_observables_by_route(ljgb_mod, canonical):
    """Records, the running averages and the last observables are those of the
    same steps, whether read after each step, at the end, through the step
    graphs (profiling, counters), or across a change of ensemble."""
    kw = dict(n=700, density=0.7, temperature=1.0, canonical=canonical, lattice=ljgb_mod.LATTICE_FCC, jitter=0.03, seed=2)
    runs = []
    for route in range(3):
        s = ljgb_mod.System(**kw)
        s.set_recording(64)
        if route == 2:
            s.counters_configure([(0, 10, 0.1, 0.0)])
        for part in (7, 1, 4):
            s.integrate(DT, part)
            if route == 1:
                s.observables()
        s.set_canonical(not canonical)
        s.integrate(DT, 3)
        runs.append((s.records(64), s.observables(), s.get_state()))
        s.close()
    for recs, o, st in runs[1:]:
        assert recs == runs[0][0] and len(recs) == 15
        assert o == runs[0][1]
        assert all(np.array_equal(a, b) for a, b in zip(st, runs[0][2]))
    # the same run on the stream-K kernel (a chosen shape)
    s = ljgb_mod.System(**kw)
    s.set_kernel_shape(0)
    s.reset_averaging()
    s.integrate(DT, 12)
    s.set_canonical(not canonical)
    s.integrate(DT, 3)
    o = s.observables()
    for k in ("U", "K", "P", "av_U_tot", "t", "step", "av_iters"):
        assert o[k] == pytest.approx(runs[0][1][k], rel=1e-6), k
    s.close()


@pytest.mark.parametrize("shape", [-1, 0])
def test_change_of_time_step_keeps_the_clock(ljgb_mod, shape):
    """The last step before a change of dt advances the clock by its own dt,
    although its observables are formed after the change."""
    s = ljgb_mod.System(n=700, density=0.7, temperature=1.0)
    s.set_kernel_shape(shape)
    s.integrate(0.004, 3)
    s.integrate(0.002, 2)
    assert s.observables()["t"] == pytest.approx(0.016, rel=1e-12)
    s.close()
