"""calculateNForces after a call in which a device-side wait ran out: such a
launch leaves its count of finished CTAs part-way.  lj_debug_reference_abi_timeout
leaves the same words behind without one.  The call that sees the flag reports
it; the next one, at other positions, gives the bits of a fresh context."""
import ctypes as C

import numpy as np
import pytest

import lj_testutil as U

pytestmark = pytest.mark.gpu

TIMEOUT = 4  # LJ_ERR_DEVICE_TIMEOUT


@pytest.mark.parametrize("n", [700, 2000, 9000])   # row kernel (all CTAs of one size, uneven), unordered pairs
@pytest.mark.parametrize("tickets", [1, 17])
def test_call_after_a_timeout(ljlib, n, tickets):
    sets = []
    for seed in (1, 2):
        pos, _, L = U.lattice_state(n, 0.7, 1.0, "fcc", 0.06, seed=seed)
        p4 = np.zeros((n, 4), np.float32)
        p4[:, :3] = pos
        sets.append(p4)
    d_pos, d_frc = C.c_void_p(), C.c_void_p()
    ljlib.allocateArray(C.byref(d_pos), n)
    ljlib.allocateArray(C.byref(d_frc), n)

    def call(p4):
        ljlib.copyArrayToDevice(d_pos, p4.ctypes.data, n)
        press, f = C.c_float(), np.zeros((n, 4), np.float32)
        ljlib.calculateNForces(d_pos, d_frc, C.byref(press), n, C.c_float(L), 1, None, C.c_float(0.1), 128, 1)
        status = ljlib.lj_reference_abi_status()
        ljlib.copyArrayFromDevice(f.ctypes.data, d_frc, 0, n)
        return status, press.value, f

    ljlib.threadExit()
    want = call(sets[1])
    assert want[0] == 0
    ljlib.threadExit()
    assert ljlib.lj_debug_reference_abi_timeout(tickets) != 0       # no buffers yet
    assert call(sets[0])[0] == 0
    assert ljlib.lj_debug_reference_abi_timeout(tickets) == 0
    assert call(sets[0])[0] == TIMEOUT
    for _ in range(2):
        status, press, f = call(sets[1])
        assert status == 0 and press == want[1] and np.array_equal(f, want[2])
    ljlib.deleteArray(d_pos)
    ljlib.deleteArray(d_frc)
    ljlib.threadExit()
