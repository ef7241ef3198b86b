"""calculateNForces on each of its pair kernels (row, unordered pairs), at the
edges of their ranges, against the FP64 oracle; the MIXED force gate (1e-5 of
max(|F|, rms F)) plus the rounding of the float results."""
import ctypes as C

import numpy as np
import pytest

import lj_testutil as U

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("n", [2, 33, 500, 2047, 8191, 8192, 8225, 12001])
def test_forces_by_range(ljgb_mod, oracle_mod, n, periodic):
    lib = ljgb_mod.load()
    pos, _, L = U.lattice_state(n, 0.6, 1.0, "fcc", 0.05, seed=n)
    p4 = np.zeros((n, 4), np.float32)
    p4[:, :3] = pos
    L = float(np.float32(L))
    d_pos, d_frc = C.c_void_p(), C.c_void_p()
    lib.allocateArray(C.byref(d_pos), n)
    lib.allocateArray(C.byref(d_frc), n)
    lib.copyArrayToDevice(d_pos, p4.ctypes.data, n)
    got = []
    for rdf in (None, np.zeros(256, np.int32), None):
        press = C.c_float()
        lib.calculateNForces(d_pos, d_frc, C.byref(press), n, C.c_float(L), int(periodic),
                             rdf.ctypes.data if rdf is not None else None, C.c_float(0.1), 128, 1)
        assert lib.lj_reference_abi_status() == 0
        f = np.zeros((n, 4), np.float32)
        lib.copyArrayFromDevice(f.ctypes.data, d_frc, 0, n)
        got.append((f, press.value))
        if rdf is not None:
            assert rdf.sum() == n * (n - 1)
    assert all(np.array_equal(f, got[0][0]) and p == got[0][1] for f, p in got)
    r = oracle_mod.f64_forces(p4[:, :3].astype(np.float64), L, periodic)
    f, press = got[0]
    assert U.force_errors(f[:, :3].astype(np.float64), r["F"])["gate_max"] <= 1.1e-5
    assert np.abs(4.0 * f[:, 3] - r["e"]).max() <= 1.1e-5 * np.abs(r["e"]).max()
    assert press == pytest.approx(r["W"] / 6, rel=2e-5, abs=1e-5 * n)
    lib.deleteArray(d_pos)
    lib.deleteArray(d_frc)
    lib.threadExit()
