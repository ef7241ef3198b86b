"""The cluster kernel (lj_cluster.cu) holds the stream for a few milliseconds at a
time: a launch has 1024 steps at most, whatever a call asks for, and the division
into launches changes no bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,canonical", [(128, 0), (512, 1)])
def test_launches_of_a_long_call(ljgb_mod, n, canonical):
    torch = pytest.importorskip("torch")
    kw = dict(n=n, density=0.3, temperature=1.2, canonical=canonical, lattice=ljgb_mod.LATTICE_FCC, jitter=0.02, seed=4)
    out = []
    for parts in ((2600,), (1000, 24, 1, 1575)):
        s = ljgb_mod.System(**kw)
        s.integrate(0.004)
        s.sync()
        c0 = s.launch_count()
        for k in parts:
            s.integrate(0.004, k)
        if len(parts) == 1:
            assert s.launch_count() - c0 == 3
        out.append((s.observables(), s.get_state()))
        s.close()
    assert out[0][0] == out[1][0] and out[0][0]["step"] == 2601
    assert all(np.array_equal(a, b) for a, b in zip(out[0][1], out[1][1]))
    # a full launch, on the device's clock
    s = ljgb_mod.System(**kw)
    st = torch.cuda.Stream()
    s.set_stream(st.cuda_stream)
    s.integrate(0.004, 64)
    best = 1e9
    for _ in range(3):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        with torch.cuda.stream(st):
            a.record()
            s.integrate(0.004, 1024)
            b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b))
    s.set_stream(None)
    s.close()
    print("1024 steps of %d: %.2f ms" % (n, best))
    assert best < 20.0
