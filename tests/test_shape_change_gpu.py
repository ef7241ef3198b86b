"""A change of the kernel shape or split cap right after a step: the step's
observables, not yet summed then, are those of a handle that reads them first."""
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("U", "K", "V", "P", "T", "t", "step", "av_U_tot", "av_p_tot", "av_iters", "Tkin_tvn")


@pytest.mark.parametrize("canonical", [0, 1])
@pytest.mark.parametrize("boxes", [1, 3])
def test_observables_across_a_change(ljgb_mod, boxes, canonical):
    cfgs = [ljgb_mod.config(n=900 + 100 * k, density=0.7, temperature=1.0, canonical=canonical,
                            lattice=ljgb_mod.LATTICE_FCC, jitter=0.03, seed=k) for k in range(boxes)]
    for change in (lambda s: s.set_kernel_shape(4), lambda s: s.set_split_cap(2), lambda s: s.set_kernel_shape(-1)):
        out = []
        for read_first in (True, False):
            s = ljgb_mod.System(batch=cfgs) if boxes > 1 else ljgb_mod.System(cfg=cfgs[0])
            s.set_kernel_shape(0)
            s.set_recording(8)
            s.integrate(0.004, 3)
            if read_first:
                s.batch_observables()
            change(s)
            out.append(([{k: o[k] for k in KEYS} for o in s.batch_observables()],
                        [s.batch_records(k, 8) for k in range(boxes)]))
            s.close()
        assert out[0] == out[1]
        assert all(len(r) == 3 for r in out[1][1])
