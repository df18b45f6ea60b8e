"""Workloads for timing the engine through its public entry points.

Every case is one call (or one short run of steps) that a program using this
package makes, with the inputs it has in hand: device tensors for the handle
API (``BHSystem``), numpy arrays for the drop-in ``api3d.compute_forces``, a
device state for the integrators.  Sizes, profiles and parameters are those of
the repository's configurations and tests: Plummer N = 4,096 (single
evaluation), Hernquist N = 2^20 (accuracy and headline), 512 systems of
1,024-65,536 bodies (batching), Plummer N = 16,384 (Parareal), N up to 2^21
(serving) and a few million (plain calls at large N).
"""
import math

import numpy as np
import torch

from hierarquicos_b200 import api3d
from hierarquicos_b200._lib import (BH_PREC_DEHNEN, BH_PREC_FP32, BH_PREC_FP64, default_params)
from hierarquicos_b200.integrate import BatchState, ForceField, symplectic_euler, verlet
from hierarquicos_b200.system import BHSystem, direct_targets, offsets_of

PRECISION = {"fp32": BH_PREC_FP32, "fp64": BH_PREC_FP64, "dehnen": BH_PREC_DEHNEN}
# flops of one cell interaction by order, and of one body-body interaction
CELL_FLOPS = {1: 20.0, 4: 60.0, 8: 140.0}
BODY_FLOPS = 20.0


def listed():
    return [
        # the smallest size of the served range and of the recorded error runs:
        # one force evaluation of a small cluster, bound by latency
        dict(name="small_1k", kind="plain", n=1024, profile="plummer", order=4, theta=0.5,
             eps=0.0, mass="equal", accel=False),
        # the single-evaluation configuration
        dict(name="plummer_4k", kind="plain", n=4096, profile="plummer", order=4, theta=0.5,
             eps=0.01, mass="equal", accel=False),
        # Parareal's coarse propagator: two symplectic-Euler steps of one window
        # with the monopole walk, the evaluation replayed from a recorded graph
        dict(name="coarse_16k", kind="euler", n=16384, profile="plummer", order=1, theta=0.8,
             eps=0.01, mass="equal", steps=2, dt=1e-2, graph=True),
        # Parareal's fine propagator: velocity-Verlet steps of a ragged batch of
        # windows / independent clusters in one batch
        dict(name="verlet_batch", kind="verlet", systems=48, lo=257, hi=16384, profile="plummer",
             order=4, theta=0.3, eps=0.01, mass="random", steps=2, dt=1e-3, graph=False),
        # an ordinary call of odd size, octupole, accelerations out
        dict(name="octupole_100k", kind="plain", n=100003, profile="sphere", order=8, theta=0.5,
             eps=0.01, mass="random", accel=True),
        # the reference's call: numpy arrays in, a new Fortran-ordered array out
        dict(name="drop_in_262k", kind="host", n=262147, profile="hernquist", order=4, theta=0.5,
             eps=0.01, mass="equal", accel=False),
        # the headline: one evaluation of a Hernquist sphere
        dict(name="hernquist_1m", kind="plain", n=1 << 20, profile="hernquist", order=4,
             theta=0.5, eps=0.01, mass="equal", accel=False),
        # a large plain call
        dict(name="sphere_5m", kind="plain", n=5000011, profile="sphere", order=4, theta=0.7,
             eps=0.01, mass="equal", accel=False),
        # many independent systems in one batched evaluation
        dict(name="batch_512", kind="batch", systems=512, lo=1024, hi=65536, profile="mixed",
             order=4, theta=0.5, eps=0.01, mass="equal", accel=False),
        # the all-FP64 walk (Parareal's FP64 propagators, accuracy runs)
        dict(name="fp64_262k", kind="plain", precision="fp64", n=262144, profile="hernquist",
             order=4, theta=0.4, eps=0.01, mass="equal", accel=False),
        # Dehnen's dual-tree method (methods 20-22)
        dict(name="dehnen_200k", kind="plain", precision="dehnen", n=200003, profile="plummer",
             order=4, theta=0.6, eps=0.01, mass="equal", accel=False),
        # the FP64 direct sum: error checks and the reference's fine propagator
        dict(name="direct_16k", kind="direct", n=16384, profile="plummer", eps=0.01,
             mass="equal", accel=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ranges; sizes log-uniform, mostly odd ones."""
    kind = rng.choice(["plain", "plain", "plain", "batch", "fp64", "dehnen", "direct", "host",
                       "euler", "verlet"])
    profile = rng.choice(["plummer", "hernquist", "sphere", "cube"])
    order = rng.choice([1, 4, 4, 8])
    theta = round(rng.uniform(0.4, 0.8), 3)
    eps = rng.choice([0.0, 0.01, 0.05])
    mass = rng.choice(["equal", "random"])
    accel = rng.random() < 0.3
    c = dict(kind=kind, profile=profile, order=order, theta=theta, eps=eps, mass=mass)
    if kind == "plain":
        c.update(n=_log_int(rng, 1000, 1 << 21), accel=accel)
        if c["n"] > (1 << 19):
            c["theta"] = round(rng.uniform(0.5, 0.8), 3)
            c["order"] = rng.choice([1, 4])
    elif kind == "batch":
        c.update(systems=_log_int(rng, 8, 256), lo=1024, hi=32768, accel=accel)
    elif kind == "fp64":
        c.update(kind="plain", precision="fp64", n=_log_int(rng, 2000, 200000), accel=accel)
    elif kind == "dehnen":
        c.update(kind="plain", precision="dehnen", n=_log_int(rng, 2000, 300000), accel=accel,
                 order=rng.choice([1, 4]))
    elif kind == "direct":
        c = dict(kind="direct", profile=profile, eps=eps, mass=mass, accel=accel,
                 n=_log_int(rng, 500, 40000))
    elif kind == "host":
        c.update(n=_log_int(rng, 1000, 1 << 19), accel=accel)
    elif kind == "euler":
        c.update(n=_log_int(rng, 1000, 40000), steps=rng.randint(1, 3), dt=1e-2, graph=True,
                 order=rng.choice([1, 4]), eps=0.01)
    else:
        c.update(systems=_log_int(rng, 4, 64), lo=257, hi=8192, steps=rng.randint(1, 3), dt=1e-3,
                 graph=False, order=rng.choice([1, 4]), eps=0.01)
    return c


# ---- inputs ----

def _sizes(case):
    """Sizes of a batch: spread over the logarithm of [lo, hi] by a fixed
    low-discrepancy sequence, so that a case's work does not depend on the seed."""
    lo, hi, k = case["lo"], case["hi"], case["systems"]
    u = (np.arange(k) * 0.6180339887498949 + 0.5 / k) % 1.0
    return np.maximum(2, np.round(np.exp(np.log(lo) + u * (np.log(hi) - np.log(lo))))).astype(int)


def _positions(profile, n, g, dev):
    def uniform(*shape):
        return torch.rand(*shape, generator=g, device=dev, dtype=torch.float64)

    if profile == "cube":
        return uniform(3, n) * 2.0 - 1.0
    u = uniform(n).clamp_(1e-12, 1.0 - 1e-12)
    if profile == "plummer":       # scale 1
        u = u * 0.999
        r = (u.pow(-2.0 / 3.0) - 1.0).rsqrt()
    elif profile == "hernquist":   # a = 1, truncated at 100 a
        s = (u * (100.0 / 101.0) ** 2).sqrt()
        r = s / (1.0 - s)
    else:                          # unit sphere of uniform density
        r = u.pow(1.0 / 3.0)
    c = uniform(n) * 2.0 - 1.0
    ph = uniform(n) * (2.0 * math.pi)
    s = (1.0 - c * c).sqrt()
    return torch.stack([r * s * ph.cos(), r * s * ph.sin(), r * c])


def _bodies(case, seed, dev="cuda"):
    """(m, q (3, N), p (3, N), offsets) on the device, from the seed alone."""
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed))
    sizes = _sizes(case) if "systems" in case else np.array([case["n"]])
    off = offsets_of(sizes)
    qs, ms = [], []
    for k, n in enumerate(sizes):
        n = int(n)
        prof = case["profile"]
        if prof == "mixed":
            prof = "plummer" if k % 2 == 0 else "sphere"
        qs.append(_positions(prof, n, g, dev))
        if case["mass"] == "equal":
            ms.append(torch.full((n,), 1.0 / n, device=dev, dtype=torch.float64))
        else:
            w = torch.rand(n, generator=g, device=dev, dtype=torch.float64) + 0.01
            ms.append(w / w.sum())
    q, m = torch.cat(qs, 1).contiguous(), torch.cat(ms)
    v = torch.randn(q.shape, generator=g, device=dev, dtype=torch.float64) * 0.3
    return m, q, v * m, off


def _params(case):
    return default_params(theta=case.get("theta", 0.5), eps=case["eps"],
                          order=case.get("order", 4), out_kind=1 if case.get("accel") else 0,
                          precision=PRECISION[case.get("precision", "fp32")])


def prepare(case, seed):
    kind = case["kind"]
    m, q, p, off = _bodies(case, seed)
    s = dict(case=case)
    if kind in ("plain", "batch"):
        x, y, z = q[0].contiguous(), q[1].contiguous(), q[2].contiguous()
        s.update(sys=BHSystem(), params=_params(case), m=m, x=x, y=y, z=z, off=off,
                 out=torch.empty(3 * m.numel(), device=m.device, dtype=torch.float64))
    elif kind == "host":
        s.update(args=[a.cpu().numpy().copy() for a in (m, q[0], q[1], q[2])])
    elif kind == "direct":
        s.update(m=m, x=q[0].contiguous(), y=q[1].contiguous(), z=q[2].contiguous())
    else:  # the integrators: a field and a scratch state stepped from (q, p)
        s.update(field=ForceField("bh", _params(case), graph=case["graph"]), q=q, p=p,
                 st=BatchState(m, q, p, off))
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "plain":
        return s["sys"].forces(s["m"], s["x"], s["y"], s["z"], s["params"], out=s["out"])
    if kind == "batch":
        return s["sys"].forces_batch(s["m"], s["x"], s["y"], s["z"], s["off"], s["params"],
                                     out=s["out"])
    if kind == "host":
        return api3d.compute_forces(*s["args"], case["theta"], 1.0, case["eps"],
                                    order=case["order"], accelerations=bool(case.get("accel")))
    if kind == "direct":
        return direct_targets(s["m"], s["x"], s["y"], s["z"], None, 1.0, case["eps"],
                              1 if case.get("accel") else 0)
    st = s["st"]
    st.q.copy_(s["q"])  # every pass steps the window's start state
    st.p.copy_(s["p"])
    if kind == "euler":
        symplectic_euler(st, s["field"], case["steps"], case["dt"])
        return [st.q, st.p]
    f = verlet(st, s["field"], case["steps"], case["dt"])
    return [st.q, st.p, f]


# ---- what a pass cannot do without ----

def _evaluations(case):
    if case["kind"] == "euler":
        return case["steps"]
    if case["kind"] == "verlet":
        return case["steps"] + 1
    return 1


def work(case):
    sizes = _sizes(case) if "systems" in case else np.array([case["n"]])
    total = float(sizes.sum())
    flops = 0.0
    for n in (float(v) for v in sizes):
        if case["kind"] == "direct":
            flops += BODY_FLOPS * n * (n - 1.0)
        elif case.get("precision") == "dehnen":
            # mutual cell-cell terms: about 170 one-sided terms per body at
            # theta 0.5, of about 130 flops (quadrupole)
            per = min(n - 1.0, 21.0 / case["theta"] ** 3)
            flops += n * per * {1: 45.0, 4: 130.0, 8: 250.0}[case["order"]]
        else:
            # accepted cells per target of the per-target walk: 2,240 at
            # N = 2^20 and theta 0.5, growing with log N and theta^-3
            cells = min(n - 1.0, 14.0 * math.log2(n) / case["theta"] ** 3)
            flops += n * cells * CELL_FLOPS[case["order"]]
    nbytes = total * (32.0 + 24.0)  # m, x, y, z in; three components out
    k = _evaluations(case)
    if case["kind"] in ("euler", "verlet"):
        nbytes = total * (8.0 + 2 * 48.0)  # m in; q and p in and out
    return dict(bytes=nbytes, flops=flops * k)


# ---- the same in 64 bits, without the engine: the softened pair sum ----

def _direct(m, q, eps, accel, off):
    """SoA blocks per system, as the engine writes them."""
    out = torch.empty(3 * m.numel(), device=m.device, dtype=torch.float64)
    for s in range(len(off) - 1):
        a, b = int(off[s]), int(off[s + 1])
        n = b - a
        x, y, z, w = q[0, a:b], q[1, a:b], q[2, a:b], m[a:b]
        f = out[3 * a:3 * b].view(3, n)
        step = max(1, min(n, (1 << 25) // n))
        for i in range(0, n, step):
            j = min(n, i + step)
            dx = x[None, :] - x[i:j, None]
            dy = y[None, :] - y[i:j, None]
            dz = z[None, :] - z[i:j, None]
            r2 = (dx * dx).addcmul_(dy, dy).addcmul_(dz, dz).add_(eps * eps)
            r2[torch.arange(j - i, device=m.device), torch.arange(i, j, device=m.device)] = math.inf
            w3 = r2.sqrt().mul_(r2).reciprocal_().mul_(w[None, :])
            f[0, i:j] = dx.mul_(w3).sum(1)
            f[1, i:j] = dy.mul_(w3).sum(1)
            f[2, i:j] = dz.mul_(w3).sum(1)
        if not accel:
            f.mul_(w[None, :])
    return out


def exact(case, seed):
    sizes = _sizes(case) if "systems" in case else np.array([case["n"]])
    if float((sizes.astype(float) ** 2).sum()) * _evaluations(case) > 1.5e11:
        return None  # too many pairs for a plain 64-bit sum
    m, q, p, off = _bodies(case, seed)
    kind = case["kind"]
    accel = bool(case.get("accel"))
    if kind in ("plain", "batch"):
        return _direct(m, q, case["eps"], accel, off)
    if kind == "direct":
        return _direct(m, q, case["eps"], accel, off).view(3, m.numel())
    if kind == "host":
        f = _direct(m, q, case["eps"], accel, off).view(3, m.numel())
        return np.asfortranarray(f.T.cpu().numpy())
    q, p, dt = q.clone(), p.clone(), case["dt"]

    def force():
        f = _direct(m, q, case["eps"], False, off)
        g = torch.empty_like(q)  # per-system blocks to rows x, y, z
        for s in range(len(off) - 1):
            a, b = int(off[s]), int(off[s + 1])
            g[:, a:b] = f[3 * a:3 * b].view(3, b - a)
        return f, g

    if kind == "euler":
        for _ in range(case["steps"]):
            _, g = force()
            p += dt * g
            q += dt * p / m
        return [q, p]
    f, g = force()
    for _ in range(case["steps"]):
        p += 0.5 * dt * g
        q += dt * p / m
        f, g = force()
        p += 0.5 * dt * g
    return [q, p, f]
