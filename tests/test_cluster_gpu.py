"""Steps of a small box in one cluster launch (lj_cluster.cu): the edges of
its rows (16 CTAs, 8 rows a warp, 8 j's a chunk), against the FP64 path with
the tolerances of tests/test_rows_gpu.py, and independence of how the steps
are divided into calls."""
import numpy as np
import pytest

import lj_testutil as U

pytestmark = pytest.mark.gpu

DT, STEPS = 0.004, 7


@pytest.mark.parametrize("canonical", [0, 1])
@pytest.mark.parametrize("boundary", [0, 1])
@pytest.mark.parametrize("N", [2, 4, 31, 32, 33, 63, 65, 127, 255, 257, 400, 449, 511, 512])
def test_cluster_steps_match_fp64(ljgb_mod, N, boundary, canonical):
    pos, vel, L = U.lattice_state(N, 0.6, 1.1, "fcc", 0.05, seed=N)
    out = []
    for prec in (0, 1):
        s = ljgb_mod.System(n=N, density=0.6, temperature=1.1, canonical=canonical, boundary=boundary, precision=prec)
        s.set_state(pos, vel)
        s.calculate_forces()
        c0 = s.launch_count()
        s.integrate(DT, STEPS)
        if prec == 0:
            assert s.launch_count() - c0 <= 2  # predictor, all steps
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


@pytest.mark.parametrize("canonical", [0, 1])
def test_cluster_steps_by_call(ljgb_mod, canonical):
    """One call, several, and host round trips give the same bits; records and
    averages have every step; a change of ensemble or dt in between holds."""
    kw = dict(n=300, density=0.7, temperature=1.0, canonical=canonical, lattice=ljgb_mod.LATTICE_FCC, jitter=0.03, seed=2)
    runs = []
    for parts in ((12,), (1, 4, 7), (1,) * 12):
        s = ljgb_mod.System(**kw)
        s.set_recording(64)
        for k in parts:
            s.integrate(DT, k)
            if len(parts) == 12:
                s.observables()
                p, v, _ = s.get_state()
                s.set_state(p, v)
        s.set_canonical(not canonical)
        s.integrate(DT, 3)
        s.integrate(DT / 2, 2)
        runs.append((s.records(64), s.observables(), s.get_state()))
        s.close()
    for recs, o, st in runs[1:]:
        assert recs == runs[0][0] and len(recs) == 17
        assert o == runs[0][1]
        assert all(np.array_equal(a, b) for a, b in zip(st, runs[0][2]))
    s = ljgb_mod.System(**kw)
    s.set_kernel_shape(0)
    s.reset_averaging()
    s.integrate(DT, 12)
    s.set_canonical(not canonical)
    s.integrate(DT, 3)
    s.integrate(DT / 2, 2)
    o = s.observables()
    for k in ("U", "K", "P", "av_U_tot", "t", "step", "av_iters"):
        assert o[k] == pytest.approx(runs[0][1][k], rel=1e-6), k
    s.close()
