"""FP64 boxes and the adjoint where the pair pass's sums cannot have their usual
size: larger squares need fewer slots.  Same pair set in another order, so
results agree to the rounding of FP64 sums: 1e-11 of the largest value bounds
that of a few thousand terms and of the ten steps' growth."""
import numpy as np
import pytest

import lj_testutil as U

pytestmark = pytest.mark.gpu


@pytest.fixture
def limit(ljlib):
    yield ljlib.lj_debug_limit_allocations
    ljlib.lj_debug_limit_allocations(-1)


def _close(a, b):
    a, b = np.asarray(a), np.asarray(b)
    assert np.abs(a - b).max() <= 1e-11 * max(1.0, np.abs(b).max())


@pytest.mark.parametrize("canonical", [0, 1])
@pytest.mark.parametrize("bytes_", [4 << 20, 1 << 20, 300_000])   # of 11 MB: sides 4, 16 and one square
def test_fp64_steps(ljgb_mod, limit, bytes_, canonical):
    n = 3000
    pos, vel, _ = U.lattice_state(n, 0.8, 1.0, "fcc", 0.04, seed=1)
    out = []
    for cap in (-1, bytes_):
        limit(cap)
        s = ljgb_mod.System(n=n, density=0.8, temperature=1.0, canonical=canonical, precision=1)
        limit(-1)
        ctas = s.tune_info()["ctas"]
        s.set_state(pos, vel)
        s.calculate_forces()
        s.integrate(0.004, 10)
        out.append((ctas, s.get_state(), s.observables()))
        s.close()
    assert out[1][0] < out[0][0]
    for a, b in zip(out[1][1], out[0][1]):
        _close(a, b)
    for k in ("U", "K", "V", "W", "T"):
        assert out[1][2][k] == pytest.approx(out[0][2][k], rel=1e-11)


def test_fp64_batch(ljgb_mod, limit):
    cfgs = [ljgb_mod.config(n=n, density=0.7, temperature=1.0, precision=1, boundary=k % 3, lattice=ljgb_mod.LATTICE_FCC,
                            jitter=0.03, seed=k) for k, n in enumerate((300, 1200, 2011))]
    out = []
    for cap in (-1, 600_000):
        limit(cap)
        s = ljgb_mod.System(batch=cfgs)
        limit(-1)
        s.integrate(0.004, 5)
        out.append(s.get_state())
        s.close()
    for a, b in zip(out[1], out[0]):
        _close(a, b)


@pytest.mark.parametrize("bytes_", [3 << 20, 300_000])
def test_adjoint(ljgb_mod, limit, bytes_):
    n = 3000
    pos, vel, _ = U.lattice_state(n, 0.8, 1.0, "fcc", 0.04, seed=2)
    out = []
    for cap in (-1, bytes_):
        limit(cap)
        a = ljgb_mod.Adjoint(n=n, density=0.8, temperature=1.0, checkpoint_every=3)
        limit(-1)
        a.set_state(pos, vel)
        out.append((a.forward(0.004, 6),) + tuple(a.backward()))
        a.close()
    for x, y in zip(out[1], out[0]):
        _close(x, y)


def test_refusal_is_reported(ljgb_mod, limit):
    limit(1000)
    for make in (lambda: ljgb_mod.System(n=3000, precision=1), lambda: ljgb_mod.Adjoint(n=3000, density=0.8)):
        with pytest.raises(ljgb_mod.LJError) as e:
            make()
        assert e.value.code == 7
