"""lj_rdf_counts where its optional buffers cannot be had (the page-locked counts,
the neighbour tiles of large boxes): the same counts by the other routes.  The
range tables, which come first, are needed and their refusal is reported."""
import numpy as np
import pytest

import lj_testutil as U

pytestmark = pytest.mark.gpu

TABLES = 3


@pytest.mark.parametrize("n", [500, 20000])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_counts_at_every_budget(ljgb_mod, ljlib, n, mode):
    pos, _, _ = U.lattice_state(n, 0.8, 1.0, "fcc", 0.05, seed=3)
    kw = dict(n=n, density=0.8, temperature=1.0)
    width = 0.05 if mode == 2 else 0.1
    want = None
    for k in [-1] + list(range(TABLES + 7)):
        s = ljgb_mod.System(**kw)
        s.set_state(pos)
        ljlib.lj_debug_fail_allocations(k)
        try:
            if 0 <= k < TABLES:
                with pytest.raises(ljgb_mod.LJError) as e:
                    s.rdf_counts(mode, 80, width)
                assert e.value.code == 7
            else:
                got = s.rdf_counts(mode, 80, width)
                want = got if want is None else want
                assert got.sum() > 0 and np.array_equal(got, want), k
        finally:
            ljlib.lj_debug_fail_allocations(-1)
        assert want is None or np.array_equal(s.rdf_counts(mode, 80, width), want)
        s.close()
