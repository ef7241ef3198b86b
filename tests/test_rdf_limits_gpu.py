"""Pair histograms with widths below FP32's range (the reciprocal width is
infinite) and with particles at one place (separation 0): every pair is past
the last bin, so the clamped histogram has all of them there and the others
none.  lj_rdf_counts and calculateNForces, over all pairs and over tiles of
neighbours."""
import ctypes as C

import numpy as np
import pytest

import lj_testutil as U

pytestmark = pytest.mark.gpu


def _state(n):
    pos, _, L = U.lattice_state(n, 0.8, 1.0, "fcc", 0.05, seed=9)
    pos[[1, n // 2, n - 1]] = pos[0]
    return pos, L


@pytest.mark.parametrize("n", [600, 16384])
def test_counts(ljgb_mod, n):
    pos, _ = _state(n)
    s = ljgb_mod.System(n=n, density=0.8, temperature=1.0)
    s.set_state(pos)
    for nb in (1, 80, 256):
        for width in (1e-42, 1e-300):
            clamped = s.rdf_counts(0, nb, width)
            assert clamped[-1] == n * (n - 1) and not clamped[:-1].any()
            assert not s.rdf_counts(1, nb, width).any()
            assert not s.rdf_counts(2, nb, width).any()
        if nb > 1:                              # the pairs at one place are ordinary pairs otherwise
            assert s.rdf_counts(0, nb, 1e-9)[0] == 12
    s.close()


@pytest.mark.parametrize("n", [600, 9000, 16384])
def test_reference_histogram(ljlib, n):
    pos, L = _state(n)
    p4 = np.zeros((n, 4), np.float32)
    p4[:, :3] = pos
    d_pos, d_frc = C.c_void_p(), C.c_void_p()
    ljlib.allocateArray(C.byref(d_pos), n)
    ljlib.allocateArray(C.byref(d_frc), n)
    ljlib.copyArrayToDevice(d_pos, p4.ctypes.data, n)
    for dr2, first in ((1e-42, 0), (1e-9, 12)):
        press, rdf = C.c_float(), np.zeros(256, np.int32)
        ljlib.calculateNForces(d_pos, d_frc, C.byref(press), n, C.c_float(L), 1, rdf.ctypes.data, C.c_float(dr2), 128, 1)
        assert ljlib.lj_reference_abi_status() == 0
        assert rdf[0] == first and rdf[255] == n * (n - 1) - first and rdf.sum() == n * (n - 1)
    ljlib.deleteArray(d_pos)
    ljlib.deleteArray(d_frc)
    ljlib.threadExit()
