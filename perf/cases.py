"""Timed cases: what programs have this library do, through its public entry points.

Every case starts from a seeded state made here with numpy (lattice sites with
jitter, Maxwell velocities), so `exact` can follow the same state in 64 bits
with torch alone.  A case's `kind` names the call a program makes:

  run      System.integrate, then the state and the observables read back
  records  System.integrate with per-step records, then the records
  io       System.step_io: a host loop that owns the state (up, step, down)
  fluct    System.integrate with the fluctuation task's counters and summed RDF
  batch    independent boxes of uneven N advanced together
  rdf      System.rdf_counts of a configuration
  adjoint  Adjoint.forward and .backward
  refabi   calculateNForces, the reference's own entry point, with its RDF

Results of the MIXED precision (FP32 pair arithmetic) are handed on in 32 bits,
what such a program stores or feeds on; those of FP64 in 64 bits.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "lennard-jones-cuda_gb300"))
import ljgb  # noqa: E402

OBS = ("K", "V", "T", "P", "U", "W")


def listed():
    return [
        # the reference's own kind of box: a few hundred gas particles, energy conserving, on the screen or in a script
        dict(name="gas_400_evn", kind="run", n=400, rho=0.05, T=1.4, tvn=0, bc=0, fp64=0, dt=0.005, steps=50),
        # an isotherm point's production: a small box at constant temperature, every step's observables kept
        dict(name="isotherm_256_tvn", kind="records", n=256, rho=0.3, T=1.4, tvn=1, bc=0, fp64=0, dt=0.004, steps=100),
        # a confined fluid of ordinary size between hard walls
        dict(name="walls_2001_evn", kind="run", n=2001, rho=0.6, T=1.2, tvn=0, bc=1, fp64=0, dt=0.004, steps=20),
        # the headline liquid, sampled every few steps
        dict(name="liquid_16384_tvn", kind="run", n=16384, rho=0.85, T=1.0, tvn=1, bc=0, fp64=0, dt=0.005, steps=4),
        # the largest single box: a solid
        dict(name="solid_131072_tvn", kind="run", n=131072, rho=1.1, T=1.0, tvn=1, bc=0, fp64=0, dt=0.004, steps=1),
        # a host program that owns the state and has each step done on the GPU
        dict(name="hostloop_4000_tvn", kind="io", n=4000, rho=0.7, T=1.1, tvn=1, bc=0, fp64=0, dt=0.005, steps=1),
        # an all-FP64 run, the yardstick of the mixed one
        dict(name="fp64_2048_evn", kind="run", n=2048, rho=0.85, T=1.0, tvn=0, bc=0, fp64=1, dt=0.005, steps=10),
        # the fluctuation task: subsystem counts and g(r) after every step
        dict(name="fluctuations_512", kind="fluct", n=512, rho=0.316, T=1.312, tvn=0, bc=0, fp64=1, dt=0.004, steps=20),
        # a parameter sweep: 256 boxes of uneven size, half of them walled, advanced together
        dict(name="sweep_256_boxes", kind="batch", boxes=256, nmin=200, nmax=4000, mix=3, dt=0.004, steps=10),
        # structure of a stored configuration
        dict(name="rdf_16384", kind="rdf", n=16384, rho=0.85, mode=0, bins=256),
        # a gradient of time-averaged energy and pressure
        dict(name="adjoint_1000", kind="adjoint", n=1000, rho=0.85, T=1.0, dt=0.005, steps=20, every=10),
        # the reference program linked against this library: one force call with its RDF
        dict(name="refabi_8000", kind="refabi", n=8000, rho=0.8, bc=0, rdf=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "run64", "records", "io", "fluct", "batch", "rdf", "adjoint", "refabi"])
    rho, T = round(rng.uniform(0.05, 0.9), 3), round(rng.uniform(0.8, 1.8), 3)
    if kind in ("run", "run64"):
        n = _log(rng, 100, 131072) if kind == "run" else _log(rng, 100, 6000)
        steps = max(1, min(50, 20000 // n)) if kind == "run" else max(1, min(20, 16000 // n))
        return dict(kind="run", n=n, rho=rho, T=T, tvn=rng.randint(0, 1), bc=rng.choice([0, 0, 0, 1, 1, 2]),
                    fp64=int(kind == "run64"), dt=rng.choice([0.004, 0.005]), steps=steps)
    if kind == "records":
        return dict(kind=kind, n=_log(rng, 100, 3000), rho=rho, T=T, tvn=rng.randint(0, 1), bc=rng.choice([0, 0, 1]),
                    fp64=0, dt=0.004, steps=rng.choice([20, 50, 100]))
    if kind == "io":
        return dict(kind=kind, n=_log(rng, 100, 40000), rho=rho, T=T, tvn=rng.randint(0, 1), bc=rng.choice([0, 0, 1]),
                    fp64=0, dt=0.005, steps=1)
    if kind == "fluct":
        return dict(kind=kind, n=_log(rng, 100, 1200), rho=rho, T=T, tvn=rng.randint(0, 1), bc=0, fp64=1, dt=0.004,
                    steps=rng.choice([10, 20]))
    if kind == "batch":
        nmin = _log(rng, 100, 400)
        return dict(kind=kind, boxes=_log(rng, 8, 256), nmin=nmin, nmax=_log(rng, nmin + 100, 4000),
                    mix=rng.randrange(1 << 30), dt=0.004, steps=10)
    if kind == "rdf":
        return dict(kind=kind, n=_log(rng, 200, 40000), rho=rho, mode=rng.randint(0, 2), bins=rng.choice([100, 200, 256]))
    if kind == "adjoint":
        return dict(kind=kind, n=_log(rng, 100, 1500), rho=rho, T=T, dt=0.004, steps=rng.choice([10, 20]),
                    every=rng.choice([5, 10, 20]))
    return dict(kind=kind, n=_log(rng, 128, 40000), rho=rho, bc=rng.choice([0, 0, 1]), rdf=rng.randint(0, 1))


# ---- seeded states -----------------------------------------------------------

def _start(n, rho, T, seed):
    """FCC sites (a random choice of them where n does not fill the cells) with
    +-0.04 sigma jitter, Maxwell velocities of zero momentum and temperature T."""
    rng = np.random.default_rng(seed)
    L = (n / rho) ** (1.0 / 3.0)
    m = math.ceil((n / 4.0) ** (1.0 / 3.0) - 1e-9)
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 1, 3)
    sites = (g + np.array([[.25, .25, .25], [.75, .75, .25], [.75, .25, .75], [.25, .75, .75]])).reshape(-1, 3)
    keep = np.sort(rng.permutation(len(sites))[:n])
    pos = sites[keep] * (L / m) + rng.uniform(-0.04, 0.04, (n, 3))
    vel = rng.normal(0.0, 1.0, (n, 3))
    vel -= vel.mean(0)
    vel *= math.sqrt(T * 3 * n / (vel ** 2).sum())
    return pos, vel, L


def _boxes(case, seed):
    """The boxes of a sweep (their sizes, rho and T by the case's mix; walls alternating)."""
    rng = np.random.default_rng(case["mix"])
    return [dict(n=int(rng.integers(case["nmin"], case["nmax"])), rho=float(rng.uniform(0.01, 1.0)),
                 T=float(rng.uniform(0.7, 2.0)), tvn=1, bc=k % 2, seed=[seed, k])
            for k in range(case["boxes"])]


def _config(c):
    return ljgb.config(n=c["n"], density=c["rho"], temperature=c.get("T", 1.0), canonical=c.get("tvn", 0),
                       boundary=c.get("bc", 0), precision=c.get("fp64", 0), lattice=ljgb.LATTICE_FCC, jitter=0.02)


COUNTERS = [(0, 20, 0.05, 0.0), (1, 20, 0.05, 0.0), (2, 20, 0.05, 0.0), (3, 20, 0.05, 0.0)]


def prepare(case, seed):
    kind, st = case["kind"], dict(case=case)
    if kind == "adjoint":
        pos, vel, _ = _start(case["n"], case["rho"], case["T"], seed)
        st["adj"] = ljgb.Adjoint(n=case["n"], density=case["rho"], temperature=case["T"], checkpoint_every=case["every"])
        st["adj"].set_state(pos, vel)
        return st
    if kind == "refabi":
        n = case["n"]
        pos, _, L = _start(n, case["rho"], 1.0, seed)
        p4 = np.zeros((n, 4), np.float32)
        p4[:, :3] = pos
        st.update(pos=torch.from_numpy(p4).cuda(), force=torch.zeros(n, 4, device="cuda"), L=float(np.float32(L)),
                  dr2=ljgb.reference_rdf_dr2(n))
        return st
    if kind == "batch":
        boxes = _boxes(case, seed)
        s = ljgb.System(batch=[_config(b) for b in boxes])
        states = [_start(b["n"], b["rho"], b["T"], b["seed"]) for b in boxes]
        pos, vel = np.concatenate([p for p, _, _ in states]), np.concatenate([v for _, v, _ in states])
    else:
        s = ljgb.System(cfg=_config(case))
        pos, vel, _ = _start(case["n"], case["rho"], case.get("T", 1.0), seed)
    s.set_state(pos, vel)
    s.calculate_forces()
    if kind == "records":
        s.set_recording(case["steps"])
    if kind == "fluct":
        s.counters_configure(COUNTERS + [(6, 20, 0.05, 3.0 * math.sqrt(case["T"]))], ring_steps=1000)
        s.rdf_accumulate(True, mode=ljgb.RDF_R_LINEAR, nbins=200, width=s.L / 400)
    s.sync()
    st.update(sys=s, pos=ljgb.pinned((s.ntotal, 3)), vel=ljgb.pinned((s.ntotal, 3)), frc=ljgb.pinned((s.ntotal, 3)))
    st["pos"][:], st["vel"][:] = pos, vel
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "adjoint":
        loss = st["adj"].forward(case["dt"], case["steps"])
        de, ds, dp, dv = st["adj"].backward()
        return dict(loss=np.float64(loss), d_eps=np.float64(de), d_sigma=np.float64(ds), d_pos=dp, d_vel=dv)
    if kind == "refabi":
        n, press = case["n"], ctypes.c_float()
        rdf = np.zeros(256, np.int32)
        ljgb.load().calculateNForces(st["pos"].data_ptr(), st["force"].data_ptr(), ctypes.byref(press), n, st["L"],
                                     int(case["bc"] == 0), rdf.ctypes.data if case["rdf"] else None, st["dr2"], 128, 1)
        return [st["force"], np.float32(press.value), rdf]
    s, pos, vel, frc = st["sys"], st["pos"], st["vel"], st["frc"]
    if kind == "rdf":
        return s.rdf_counts(case["mode"], case["bins"], s.L / 2 / case["bins"] if case["mode"] == 2 else None).astype(np.int64)
    if kind == "io":
        o = s.step_io(case["dt"], case["steps"], pos, vel, pos, vel, frc)
        return _handed(case, pos, vel, frc, np.array([o[k] for k in OBS]))
    s.integrate(case["dt"], case["steps"])
    if kind == "records":
        r = s.records(case["steps"])
        return {k: np.array([x[k] for x in r], np.float32) for k in OBS}
    if kind == "batch":
        s.get_state_into(pos, vel, frc)
        return _handed(case, pos, vel, frc, np.array([[o[k] for k in OBS] for o in s.batch_observables()]))
    o = s.get_state_observables_into(pos, vel, frc)
    out = _handed(case, pos, vel, frc, np.array([o[k] for k in OBS]))
    if kind == "fluct":
        out["counts"] = s.counters_read()
        out["rdf"] = s.rdf_accumulated(reset=True)[0].astype(np.int64)
    return out


def _handed(case, pos, vel, frc, obs):
    t = np.float64 if case.get("fp64") else np.float32
    return dict(pos=np.asarray(pos).astype(t), vel=np.asarray(vel).astype(t), force=np.asarray(frc).astype(t),
                obs=obs.astype(t))


# ---- what a pass cannot do without ----------------------------------------------

# Flops of one unordered pair evaluated once: separation and r^2 (8), reciprocal
# and powers (5), force factor (3), both particles' forces (12), energies and
# virials (8).  The adjoint's reverse pass adds the Hessian-vector product and
# the sigma derivatives.
PAIR, PAIR_HVP, PAIR_RDF = 36, 100, 12


def work(case):
    kind = case["kind"]
    if kind == "batch":
        mean = [(case["nmin"] + case["nmax"]) / 2, (case["nmin"] ** 2 + case["nmin"] * case["nmax"] + case["nmax"] ** 2) / 3]
        return dict(bytes=case["boxes"] * mean[0] * (72 + 72), flops=case["boxes"] * mean[1] / 2 * PAIR * case["steps"])
    n = case["n"]
    pairs = n * (n - 1) / 2
    if kind == "adjoint":
        return dict(bytes=n * (48 + 48 + case["steps"] * 72), flops=pairs * case["steps"] * (PAIR + PAIR + PAIR_HVP))
    if kind == "refabi":
        return dict(bytes=n * 32, flops=pairs * (PAIR + PAIR_RDF * case["rdf"]))
    if kind == "rdf":
        return dict(bytes=n * 24, flops=pairs * PAIR_RDF)
    rdf = PAIR_RDF if kind == "fluct" else 0
    return dict(bytes=n * (72 + (0 if kind == "records" else 72)), flops=pairs * case["steps"] * (PAIR + rdf))


# ---- the same in 64 bits, with torch alone ----------------------------------------

def _pair_sums(x, L, periodic):
    """Forces, per-particle sums of r^-12 and r^-6 (eps = sigma = 1), rows in slabs."""
    n = len(x)
    F, A, B = torch.zeros_like(x), x.new_zeros(n), x.new_zeros(n)
    step = max(1, min(n, (1 << 26) // n))
    for i in range(0, n, step):
        d = x[i:i + step, None] - x[None]
        if periodic:
            d -= L * torch.round(d / L)
        r2 = (d * d).sum(-1)
        r2[torch.arange(len(r2)), torch.arange(i, i + len(r2))] = math.inf
        r6 = r2.pow(-3)
        F[i:i + step] = ((48 * r6 * r6 - 24 * r6) / r2)[..., None].mul(d).sum(1)
        A[i:i + step], B[i:i + step] = (r6 * r6).sum(1), r6.sum(1)
    return F, A, B


def _follow(x, v, L, c, dt, steps):
    """The state and, for each step, the observables of `steps` steps."""
    n, periodic, obs = len(x), c["bc"] == 0, []
    F = _pair_sums(x, L, periodic)[0]
    for _ in range(steps):
        x = x + dt * v + 0.5 * dt * dt * F
        F0 = F
        F, A, B = _pair_sums(x, L, periodic)
        tf = 0.5 * (F0 + F)
        if c["tvn"]:
            tv = v + 0.5 * dt * tf
            chi = torch.sqrt(c["T"] * 3 * n / (tv * tv).sum())
            v = (2 * chi - 1) * v + chi * dt * tf
        else:
            v = v + dt * tf
        if periodic:
            x = torch.where(x < 0, x + L, x)
            x = torch.where(x > L, x - L, x)
        elif c["bc"] == 1:
            v = torch.where(((x < 0) & (v < 0)) | ((x > L) & (v > 0)), -v, v)
        K, V, W = 0.5 * (v * v).sum(), 2 * (A - B).sum(), (48 * A - 24 * B).sum()
        T = 2 * K / 3 / n
        obs.append(torch.stack([K, V, T, (W / 6 + n * T) * c["rho"] / n, K + V, W]))
    return x, v, F, torch.stack(obs)


def _on_gpu(a):
    return torch.from_numpy(np.ascontiguousarray(a)).double().cuda()


def exact(case, seed):
    kind = case["kind"]
    if kind == "rdf":
        return None
    if kind == "adjoint":
        return _exact_gradient(case, seed)
    if kind == "refabi":
        pos, _, L = _start(case["n"], case["rho"], 1.0, seed)
        F, A, B = _pair_sums(_on_gpu(pos.astype(np.float32)), float(np.float32(L)), case["bc"] == 0)
        return [torch.cat([F, (A - B)[:, None]], 1), float((48 * A - 24 * B).sum()) / 6, None]
    if kind == "batch":
        got = []
        for b in _boxes(case, seed):
            pos, vel, L = _start(b["n"], b["rho"], b["T"], b["seed"])
            got.append(_follow(_on_gpu(pos), _on_gpu(vel), L, b, case["dt"], case["steps"]))
        return dict(pos=torch.cat([g[0] for g in got]), vel=torch.cat([g[1] for g in got]),
                    force=torch.cat([g[2] for g in got]), obs=torch.stack([g[3][-1] for g in got]))
    pos, vel, L = _start(case["n"], case["rho"], case["T"], seed)
    x, v, F, obs = _follow(_on_gpu(pos), _on_gpu(vel), L, case, case["dt"], case["steps"])
    if kind == "records":
        return {k: obs[:, j] for j, k in enumerate(OBS)}
    out = dict(pos=x, vel=v, force=F, obs=obs[-1])
    if kind == "fluct":
        out.update(counts=None, rdf=None)
    return out


def _exact_gradient(case, seed):
    """Autograd through the forward pass: loss = mean over steps of V/N + P."""
    pos, vel, L = _start(case["n"], case["rho"], case["T"], seed)
    n, dt = case["n"], case["dt"]
    x0, v0 = _on_gpu(pos).requires_grad_(), _on_gpu(vel).requires_grad_()
    eps, sig = (torch.ones((), dtype=torch.float64, device="cuda", requires_grad=True) for _ in range(2))
    own = torch.eye(n, dtype=torch.bool, device="cuda")

    def sums(x):
        d = x[:, None] - x[None]
        d = d - L * torch.round(d.detach() / L)
        r2 = (d * d).sum(-1).masked_fill(own, 1.0)
        s6 = ((sig * sig / r2) ** 3).masked_fill(own, 0.0)
        u = 4 * eps * (12 * s6 * s6 - 6 * s6)
        return ((u / r2)[..., None] * d).sum(1), 2 * eps * (s6 * s6 - s6).sum(), u.sum()

    x, v, loss = x0, v0, 0.0
    F, _, _ = sums(x)
    for _ in range(case["steps"]):
        x = x + dt * v + 0.5 * dt * dt * F
        shift = torch.where(x < 0, L, 0.0) - torch.where(x > L, L, 0.0)
        x, v = x + shift, v + 0.5 * dt * F
        F, V, W = sums(x)
        v = v + 0.5 * dt * F
        T = (v * v).sum() / 3 / n
        loss = loss + (V / n + (W / 6 + n * T) * case["rho"] / n) / case["steps"]
    de, ds, dp, dv = torch.autograd.grad(loss, [eps, sig, x0, v0])
    return dict(loss=loss.detach(), d_eps=de, d_sigma=ds, d_pos=dp, d_vel=dv)
