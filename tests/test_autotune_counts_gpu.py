"""lj_autotune steps the system to time it and puts the state back; its steps are
no samples of the counters, the summed RDF or the records either."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [400, 1500, 9000])
def test_trials_are_not_counted(ljgb_mod, n):
    out = []
    for tune in (False, True):
        s = ljgb_mod.System(n=n, density=0.6, temperature=1.0, canonical=1, lattice=ljgb_mod.LATTICE_FCC, jitter=0.03)
        s.set_recording(16)
        s.counters_configure([(0, 10, 0.1, 0.0), (3, 10, 0.1, 0.0)], ring_steps=16)
        s.counters_set_interval(2)
        s.rdf_accumulate(True, mode=2, nbins=40, width=0.05)
        s.integrate(0.004, 5)
        if tune:
            s.autotune()
        s.integrate(0.004, 3)
        c = s.counters_read()
        r, samples = s.rdf_accumulated()
        out.append((c, samples, int(r.sum()), len(s.records(16)), s.observables()["step"]))
        s.close()
    assert len(out[0][0]) == 4 and out[0][1] == 8 and out[0][3] == 8
    assert out[1][1:] == out[0][1:]
    # the shape may differ from then on: counts agree but for particles at an edge
    assert out[1][0].shape == out[0][0].shape and np.abs(out[1][0] - out[0][0]).max() <= 2
