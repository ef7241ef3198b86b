"""lj_step on a stream that a caller is capturing is refused, and leaves the handle
as it was: the next step outside the capture is that of a twin."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,precision,boxes", [(300, 0, 1), (900, 0, 1), (9000, 0, 1), (600, 1, 1), (400, 0, 3)])
@pytest.mark.parametrize("before", [0, 3])
@pytest.mark.parametrize("dt", [0.004, 0.002])
def test_step_after_a_refused_capture(ljgb_mod, n, precision, boxes, before, dt):
    torch = pytest.importorskip("torch")
    cfgs = [ljgb_mod.config(n=n + k, density=0.7, temperature=1.0, precision=precision, canonical=1,
                            lattice=ljgb_mod.LATTICE_FCC, jitter=0.03, seed=k) for k in range(boxes)]
    st = torch.cuda.Stream()
    out = []
    for capture in (False, True):
        s = ljgb_mod.System(batch=cfgs) if boxes > 1 else ljgb_mod.System(cfg=cfgs[0])
        s.set_stream(st.cuda_stream)
        if before:
            s.integrate(0.004, before)
        p, v, _ = s.get_state()
        s.set_state(p * 1.0001, v)
        if capture:
            g = torch.cuda.CUDAGraph()
            with pytest.raises(ljgb_mod.LJError):
                with torch.cuda.graph(g, stream=st, capture_error_mode="thread_local"):
                    s.integrate(dt, 2)
            torch.cuda.synchronize()
            del g
        s.integrate(dt, 2)
        out.append((s.get_state(), s.batch_observables()))
        s.set_stream(None)
        s.close()
    assert all(np.array_equal(a, b) for a, b in zip(out[0][0], out[1][0]))
    assert out[0][1] == out[1][1]
