"""The counting launch at the edges of its CTAs (128 particles) and of its
ring (one row more than is read): counts are whole numbers, so equal to the
numpy restatement of the reference's counting functions (oracle/tasks.py)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [32, 127, 128, 129, 300])
def test_counts_through_a_wrapping_ring(ljgb_mod, n):
    import tasks
    s = ljgb_mod.System(n=n, density=0.1, temperature=1.3)
    s.counters_configure([(0, 19, 0.05, 0.0), (3, 19, 0.05, 0.0), (4, 20, 0.05, 2.5)], ring_steps=3)
    expect = []

    def step(k):
        for _ in range(k):
            s.integrate(0.004)
            p, v, _ = s.get_state()
            expect.append(np.concatenate([tasks.subsystem_counts(p, s.L, 0.05, 0),
                                          tasks.subsystem_counts(p, s.L, 0.05, 3),
                                          tasks.velocity_counts(v, 2.5, 0.05, 0)]))

    got = []
    for k in (2, 3, 1, 3, 3):           # the fourth row and the first one follow each other
        step(k)
        got.append(s.counters_read())
        assert got[-1].shape[0] == k
    assert np.array_equal(np.concatenate(got), np.array(expect))
