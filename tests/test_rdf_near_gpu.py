"""Short-ranged histograms of large boxes, which leave out pairs of far tiles:
counts are whole numbers, so equal to the exact emulation (periodic boxes), and
to the full pass elsewhere -- the same box with more bins, which reach too far
for tiles to be left out."""
import ctypes as C

import numpy as np
import pytest

import lj_testutil as U

pytestmark = pytest.mark.gpu


def _positions(kind, N, rho, seed):
    pos, vel, L = U.lattice_state(N, rho, 1.0, "fcc", 0.05, seed=seed)
    rng = np.random.default_rng(seed)
    if kind == "shuffled":       # no order in memory to help
        pos = pos[rng.permutation(N)]
    elif kind == "droplet":      # nearly everything in a few cells, across the period's edge
        pos = (0.02 * pos + np.array([0.99, 0.5, 0.0]) * L) % L
        pos[:7] = rng.uniform(0, L, (7, 3))
    return pos, vel, L


@pytest.mark.parametrize("kind", ["lattice", "shuffled", "droplet"])
@pytest.mark.parametrize("N", [16384, 16385, 20001])
def test_near_tiles_match_the_emulation(ljgb_mod, oracle_mod, N, kind):
    rho = 0.3
    pos, vel, L = _positions(kind, N, rho, N)
    s = ljgb_mod.System(n=N, density=rho)
    s.set_state(pos, vel)
    q, ks = oracle_mod.emu_fixed(pos, L), L / 4294967296.0
    k2 = np.float32(ks * ks)
    for nb, w in ((64, 0.3), (1, 1.7)):
        for mode in (0, 1):
            assert np.array_equal(s.rdf_counts(mode, nb, w), oracle_mod.emu_rdf_r2(q, k2, np.float32(1.0 / w), nb, mode))
    nb, dr = 60, 0.1
    rmax = nb * dr
    assert np.array_equal(s.rdf_counts(2, nb, dr),
                          oracle_mod.emu_rdf_r(q, k2, np.float32(1.0 / dr), np.float32(rmax * rmax), nb))
    s.close()


@pytest.mark.parametrize("boundary", [0, 1, 2])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_near_tiles_match_the_full_pass(ljgb_mod, boundary, mode):
    N, rho, nb, w = 17001, 0.4, 40, 0.2
    pos, vel, L = _positions("shuffled", N, rho, 3)
    s = ljgb_mod.System(n=N, density=rho, boundary=boundary)
    s.set_state(pos, vel)
    s.integrate(0.002, 3)
    near, full = s.rdf_counts(mode, nb, w), s.rdf_counts(mode, 4000, w)
    k = nb - 1 if mode == 0 else nb          # the clamped mode's last bin holds the rest
    assert np.array_equal(near[:k], full[:k]) and near[:k].sum() > 0
    if mode == 0:
        assert near.sum() == full.sum() == N * (N - 1)
    s.close()


@pytest.mark.parametrize("n", [16385, 20001])
def test_reference_call_counts(ljgb_mod, oracle_mod, n):
    lib = ljgb_mod.load()
    pos, _, L = _positions("shuffled", n, 0.5, n)
    p4, L = np.zeros((n, 4), np.float32), float(np.float32(L))
    p4[:, :3] = pos
    d_pos, d_frc, rdf, press = C.c_void_p(), C.c_void_p(), np.zeros(256, np.int32), C.c_float()
    lib.allocateArray(C.byref(d_pos), n)
    lib.allocateArray(C.byref(d_frc), n)
    lib.copyArrayToDevice(d_pos, p4.ctypes.data, n)
    ks = L / 4294967296.0
    want = oracle_mod.emu_rdf_r2(oracle_mod.emu_fixed(p4[:, :3].astype(np.float64), L), np.float32(ks * ks),
                                 np.float32(1.0) / np.float32(0.1), 256, 0)
    for _ in range(2):
        lib.calculateNForces(d_pos, d_frc, C.byref(press), n, C.c_float(L), 1, rdf.ctypes.data, C.c_float(0.1), 128, 1)
        assert lib.lj_reference_abi_status() == 0 and np.array_equal(rdf, want)
    lib.calculateNForces(d_pos, d_frc, C.byref(press), n, C.c_float(L), 0, rdf.ctypes.data, C.c_float(0.1), 128, 1)
    assert rdf.sum() == n * (n - 1)
    lib.deleteArray(d_pos)
    lib.deleteArray(d_frc)
    lib.threadExit()
