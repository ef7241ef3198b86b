"""Profiled steps go through captured step graphs (the events need nodes);
others go to the stream directly.  Both queue the same launches, so state,
records, counters and histogram agree bit for bit, for each of the pair kernels
and with a change of route in between.  Boxes of up to 512 particles take the
row kernel when profiled, or counted, or with a summed histogram."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DT = 0.004
COUNTERS = [(0, 10, 0.1, 0.0), (3, 10, 0.1, 0.0)]


def _run(ljgb, cfgs, route, extras):
    s = ljgb.System(batch=cfgs) if len(cfgs) > 1 else ljgb.System(cfg=cfgs[0])
    s.set_recording(32)
    if extras:
        s.counters_configure(COUNTERS)
        s.rdf_accumulate(True, mode=2, nbins=50, width=0.05)
    for k, steps in enumerate((3, 1, 4)):
        if route == "mixed":
            s.profile(k % 2 == 0)
        else:
            s.profile(route == "graph")
        s.integrate(DT, steps)
    prof = s.profile_read()
    got = [s.get_state(), s.batch_observables(), [s.batch_records(b, 32) for b in range(len(cfgs))]]
    if extras:
        got += [s.counters_read(), s.rdf_accumulated()]
    s.set_canonical(not cfgs[0].canonical)
    s.integrate(DT, 2)
    got.append(s.get_state())
    s.close()
    return got, prof


def _same(a, b):
    if isinstance(a, (list, tuple)):
        return len(a) == len(b) and all(_same(x, y) for x, y in zip(a, b))
    if isinstance(a, np.ndarray):
        return np.array_equal(a, b)
    return a == b


@pytest.mark.parametrize("canonical", [0, 1])
@pytest.mark.parametrize("n,precision,boundary,extras", [
    (300, 0, 0, True), (700, 0, 0, False), (700, 0, 1, True), (700, 0, 2, False),   # row kernel; open: phase by phase
    (9000, 0, 0, False), (9000, 0, 1, True),                                        # unordered pairs
    (600, 1, 0, False), (600, 1, 0, True), (600, 1, 1, True)])                      # FP64
def test_graphs_give_the_same_bits(ljgb_mod, n, precision, boundary, extras, canonical):
    cfgs = [ljgb_mod.config(n=n, density=0.6, temperature=1.1, canonical=canonical, boundary=boundary,
                            precision=precision, lattice=ljgb_mod.LATTICE_FCC, jitter=0.03, seed=3)]
    want, _ = _run(ljgb_mod, cfgs, "plain", extras)
    for route in ("graph", "mixed"):
        got, prof = _run(ljgb_mod, cfgs, route, extras)
        assert _same(got, want), route
        if route == "graph":
            assert prof["steps"] >= 1 and prof["step_ms"] > 0


def test_graphs_of_a_batch(ljgb_mod):
    cfgs = [ljgb_mod.config(n=300 + 157 * k, density=0.5, temperature=1.1, canonical=1, boundary=k % 2,
                            lattice=ljgb_mod.LATTICE_FCC, jitter=0.03, seed=k) for k in range(4)]
    want, _ = _run(ljgb_mod, cfgs, "plain", False)
    for route in ("graph", "mixed"):
        assert _same(_run(ljgb_mod, cfgs, route, False)[0], want), route
