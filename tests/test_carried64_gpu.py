"""FP64 steps of periodic boxes carry the next step's drift in the shadow.
Whatever comes between two steps -- a change of dt, new velocities, new
positions, forces, a histogram, another boundary and back, the trajectory is
that of the FP64 oracle stepping the same states; sums differ in order only, so
over a few steps at 1e-10 of the box."""
import numpy as np
import pytest

import lj_testutil as U

pytestmark = pytest.mark.gpu

TOL = 1e-10


@pytest.mark.parametrize("tvn", [0, 1], ids=["evn", "tvn"])
@pytest.mark.parametrize("N", [31, 33, 300, 1601])
def test_what_comes_between_steps(ljgb_mod, oracle_mod, N, tvn):
    rho, T0 = 0.4, 1.2
    pos, vel, L = U.lattice_state(N, rho, T0, "fcc", 0.05, seed=N)
    s = ljgb_mod.System(n=N, density=rho, temperature=T0, canonical=tvn, precision=ljgb_mod.PREC_FP64)
    s.set_state(pos, vel)
    s.calculate_forces()
    ref = [pos, vel]

    def follow(dt, steps, bc=0):
        """The oracle from the state read back last, against the GPU."""
        o = oracle_mod.F64System(ref[0], ref[1], L, rho, T0, bool(tvn), bc, nthreads=4)
        for _ in range(steps):
            o.step(dt)
        s.integrate(dt, steps)
        p, v, _ = s.get_state()
        assert np.abs(p - o.pos).max() <= TOL * L and np.abs(v - o.vel).max() <= TOL * np.abs(o.vel).max()
        ob = s.observables()
        for key in ("K", "V", "U", "P"):
            assert ob[key] == pytest.approx(getattr(o, key), rel=1e-9, abs=1e-9 * N)
        ref[:] = [p, v]

    follow(0.002, 3)
    follow(0.001, 2)                                  # another dt
    s.rdf_counts(ljgb_mod.RDF_R2_CLAMP, 64, 0.1)      # a pass of its own over the shadow
    follow(0.001, 1)
    ref[1] = 0.5 * ref[1]
    s.set_state(None, ref[1])                         # new velocities
    follow(0.001, 2)
    s.set_state(pos, None)                            # new positions
    s.calculate_forces()
    ref[0] = pos
    follow(0.002, 2)
    for bc in (1, 0):                                 # another boundary and back
        s.set_boundary(bc)
        s.calculate_forces()
        follow(0.002, 2, bc)
        # a histogram of every step: walled boxes then rebuild their frames in
        # between, periodic steps leave its shadow behind
        s.rdf_accumulate(True, mode=ljgb_mod.RDF_R2_CLAMP, nbins=64, width=0.1)
        follow(0.002, 1, bc)
        counts, samples = s.rdf_accumulated(reset=True)
        assert samples == 1 and np.array_equal(counts, s.rdf_counts(ljgb_mod.RDF_R2_CLAMP, 64, 0.1))
        s.rdf_accumulate(False)
        follow(0.002, 1, bc)
