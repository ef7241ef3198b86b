"""A box in the unordered-pair kernel's range without the memory for its sums:
the box is created all the same and steps by the stream-K kernel (two launches
a TVN step instead of three).  Everything else a creation allocates comes
first, so what the sums may lack is the sums' own."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OOM, DT = 7, 0.004
KW = dict(n=9000, density=0.8, temperature=1.0, canonical=1, jitter=0.03, seed=5)
NEWTON_BUFFERS = 5


def _launches(s, steps=3):
    s.integrate(DT)
    c0 = s.launch_count()
    s.integrate(DT, steps)
    return (s.launch_count() - c0) // steps


def test_creation_without_the_sums(ljgb_mod, ljlib):
    want = ljgb_mod.System(**KW, lattice=ljgb_mod.LATTICE_FCC)
    assert _launches(want) == 3
    o = want.observables()
    want.close()
    cfg = ljgb_mod.config(**KW, lattice=ljgb_mod.LATTICE_FCC)
    made = []
    for k in range(200):
        h = ljgb_mod._P()
        ljlib.lj_debug_fail_allocations(k)
        rc = ljlib.lj_create(C.byref(cfg), C.byref(h))
        ljlib.lj_debug_fail_allocations(-1)
        assert rc in (0, OOM)
        if rc == 0:
            ljlib.lj_destroy(h)
            made.append(k)
            if len(made) > NEWTON_BUFFERS:
                break
    first = made[0]
    assert first >= 15 and made == list(range(first, first + NEWTON_BUFFERS + 1))
    for k, per_step in [(first + m, 2) for m in range(NEWTON_BUFFERS)] + [(first + NEWTON_BUFFERS, 3)]:
        ljlib.lj_debug_fail_allocations(k)
        s = ljgb_mod.System(cfg=cfg)
        ljlib.lj_debug_fail_allocations(-1)
        assert _launches(s) == per_step, k
        for key in ("U", "K", "P", "t"):
            assert s.observables()[key] == pytest.approx(o[key], rel=1e-6), (k, key)
        if k == first:                          # the memory is there again
            s.set_kernel_shape(-1)
            assert _launches(s) == 3
        s.close()


def test_a_chosen_shape_holds_no_sums(ljgb_mod):
    torch = pytest.importorskip("torch")
    kw = dict(n=60000, density=0.8, temperature=1.0, canonical=1, lattice=ljgb_mod.LATTICE_FCC)
    used = []
    for hint in (0, 128):
        torch.cuda.synchronize()
        free0 = torch.cuda.mem_get_info()[0]
        s = ljgb_mod.System(**kw, block_hint=hint)
        used.append(free0 - torch.cuda.mem_get_info()[0])
        assert _launches(s) == (2 if hint else 3)
        s.set_kernel_shape(-1)
        assert _launches(s) == 3
        s.close()
    assert used[0] - used[1] >= 100 << 20       # 2.3 KB a particle at this size
