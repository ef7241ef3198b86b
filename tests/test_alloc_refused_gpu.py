"""Allocations that CUDA itself refuses: requests larger than the device's whole
memory, which fail at once and take nothing.  (lj_debug_fail_allocations, which
the other out-of-memory tests use, refuses before CUDA is called, so it cannot
show what a refusal leaves behind in the runtime.)  The handle works on as if
the call had not been made."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OOM = 7
HUGE = 2 ** 31 - 1


def test_step_after_a_refused_allocation(ljgb_mod):
    cfgs = [ljgb_mod.config(n=300 + k, density=0.7, temperature=1.0, lattice=ljgb_mod.LATTICE_FCC) for k in range(4)]
    a, b = ljgb_mod.System(batch=cfgs), ljgb_mod.System(batch=cfgs)
    with pytest.raises(ljgb_mod.LJError) as e:
        a.set_recording(HUGE)               # 4 rings of 2^31 records of 112 bytes: 0.96 TB
    assert e.value.code == OOM
    for s in (a, b):
        s.integrate(0.004, 3)
    assert all(np.array_equal(x, y) for x, y in zip(a.get_state(), b.get_state()))
    a.close()
    b.close()


def test_creation_after_a_refused_allocation(ljgb_mod):
    adj = ljgb_mod.Adjoint(n=2000, density=0.7, temperature=1.0, checkpoint_every=1)
    with pytest.raises(ljgb_mod.LJError) as e:
        adj.forward(0.004, HUGE)            # 2^31 checkpoints of 145 KB: 0.3 PB
    assert e.value.code == OOM
    s = ljgb_mod.System(n=500, density=0.7, temperature=1.0)
    s.integrate(0.004, 2)
    assert np.isfinite(s.observables()["U"])
    s.close()
    assert np.isfinite(adj.forward(0.004, 2))
    adj.close()
