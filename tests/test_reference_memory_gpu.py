"""calculateNForces where the unordered-pair sums cannot be had: the call goes
through on the stream-K kernel (and the histogram over all pairs), with the
forces of the FP64 oracle at the MIXED gate (1e-5 of max(|F|, rms F), and a
tenth of it for the rounding of the float results) and the same histogram."""
import ctypes as C

import numpy as np
import pytest

import lj_testutil as U

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8192, 9001, 20000])
def test_call_without_the_sums(ljlib, oracle_mod, n):
    pos, _, L = U.lattice_state(n, 0.8, 1.0, "fcc", 0.05, seed=n)
    p4 = np.zeros((n, 4), np.float32)
    p4[:, :3] = pos
    L = float(np.float32(L))
    d_pos, d_frc = C.c_void_p(), C.c_void_p()
    ljlib.allocateArray(C.byref(d_pos), n)
    ljlib.allocateArray(C.byref(d_frc), n)
    ljlib.copyArrayToDevice(d_pos, p4.ctypes.data, n)
    got = []
    for limit in (-1, 400 * n):           # 160 bytes a particle for stream-K, 1 KB and more for the sums
        ljlib.threadExit()
        press, rdf, f = C.c_float(), np.zeros(256, np.int32), np.zeros((n, 4), np.float32)
        ljlib.lj_debug_limit_allocations(limit)
        ljlib.calculateNForces(d_pos, d_frc, C.byref(press), n, C.c_float(L), 1, rdf.ctypes.data, C.c_float(0.1), 128, 1)
        ljlib.lj_debug_limit_allocations(-1)
        assert ljlib.lj_reference_abi_status() == 0
        ljlib.copyArrayFromDevice(f.ctypes.data, d_frc, 0, n)
        got.append((f, press.value, rdf))
    (f0, p0, h0), (f1, p1, h1) = got
    assert not np.array_equal(f0, f1)                      # another kernel's rounding
    assert np.array_equal(h0, h1) and h0.sum() == n * (n - 1)
    r = oracle_mod.f64_forces(p4[:, :3].astype(np.float64), L, True)
    for f, p, _ in got:
        assert U.force_errors(f[:, :3].astype(np.float64), r["F"])["gate_max"] <= 1.1e-5
        assert p == pytest.approx(r["W"] / 6, rel=2e-5)
    # nothing at all: the call still reports it
    ljlib.threadExit()
    ljlib.lj_debug_limit_allocations(16)
    ljlib.calculateNForces(d_pos, d_frc, C.byref(press), n, C.c_float(L), 1, None, C.c_float(0.1), 128, 1)
    ljlib.lj_debug_limit_allocations(-1)
    assert ljlib.lj_reference_abi_status() == 7
    ljlib.deleteArray(d_pos)
    ljlib.deleteArray(d_frc)
    ljlib.threadExit()
