"""The workloads whose speed is measured, each through the public Python binding (``pawan_b200.capi``).

Six kinds of call, all of them what a vortex-particle program does with the library:

* ``step``      - upload the wakes, advance them some time steps on the device, download them (what the C++ drop-in's
                  integrators do per call): RK4 / RK3 / Euler, one system or a batch of independent ones, FP32C or FP64,
                  optionally split positions and a uniform inflow.
* ``solve``     - one rate evaluation (velocity and dalpha/dt) of the resident particles, downloaded; Gaussian or
                  high-order kernel, FP32C or FP64.
* ``diagnose``  - the conserved-quantity record of the resident particles.
* ``probe``     - the velocity induced at arbitrary points (a rotor's airstations, a survey plane).
* ``field``     - the vorticity field at the particles, which the strength solve builds its matrix from.
* ``surrogate`` - one rate evaluation by the octree surrogate, its sampled check included.

An FP32C context computes its pair terms in FP32, so a program that keeps its results keeps them in float32: that is
the type they are returned in here.  FP64 contexts, probes and the vorticity field (FP64 in both modes) return float64.
"""
import math

import numpy as np
import torch

from pawan_b200 import capi, cases as layouts

NU = 1e-4
# beyond this many ordered pairs the plain FP64 evaluation of exact() would take too long
EXACT_PAIRS = 2.5e10


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest ring of the fixtures, one RK4 step per call: the drop-in's step() in PAWAN's own time loop, where
        # transfers, launches and an almost empty device count
        {"name": "step_ring_1000", "kind": "step", "layout": "stations", "n": 1000, "precision": "fp32c",
         "scheme": "rk4", "steps": 1},
        # the 5000-particle single ring, ten RK4 steps on the device between two downloads
        {"name": "steps_ring_5000", "kind": "step", "layout": "stations", "n": 5000, "precision": "fp32c",
         "scheme": "rk4", "steps": 10},
        # the same ring in the FP64 mode, for a parity run against PAWAN
        {"name": "step_ring_5000_fp64", "kind": "step", "layout": "stations", "n": 5000, "precision": "fp64",
         "scheme": "rk4", "steps": 1},
        # a batch of independent rings of uneven sizes, one RK4 step: a parameter sweep in one context
        {"name": "step_batch_16_rings", "kind": "step", "layout": "uneven", "count": 16, "nmin": 2000, "nmax": 40000,
         "precision": "fp32c", "scheme": "rk4", "steps": 1},
        # a rotor's tip-vortex wake, dense filaments with split positions and inflow, one RK3 step per shedding
        {"name": "step_rotor_wake_rk3", "kind": "step", "layout": "rotor", "per_blade": 199, "sheds": 31,
         "precision": "fp32c", "scheme": "rk3", "steps": 1, "split": True, "inflow": True},
        # one rate evaluation of the 1M-particle ring: the headline size
        {"name": "solve_ring_1m", "kind": "solve", "layout": "gauss", "n": 1000000, "precision": "fp32c",
         "kernel": "gaussian"},
        # the same geometry in the FP64 mode, a ragged size
        {"name": "solve_ring_60001_fp64", "kind": "solve", "layout": "gauss", "n": 60001, "precision": "fp64",
         "kernel": "gaussian"},
        # PAWAN's second regularisation kernel
        {"name": "solve_highorder_60000", "kind": "solve", "layout": "gauss", "n": 60000, "precision": "fp32c",
         "kernel": "highorder"},
        # the diagnostics record written after every step
        {"name": "diagnose_ring_100000", "kind": "diagnose", "layout": "gauss", "n": 100000, "precision": "fp32c",
         "kernel": "gaussian"},
        # the inflow at a rotor's airstations (4 blades x 100) from a large wake
        {"name": "probe_400_of_100000", "kind": "probe", "layout": "gauss", "n": 100000, "points": 400,
         "precision": "fp32c", "kernel": "gaussian"},
        # the vorticity field of the strength solve
        {"name": "field_ring_30000", "kind": "field", "layout": "gauss", "n": 30000, "precision": "fp32c",
         "kernel": "gaussian"},
        # two coaxial rings of 1M particles together, by the octree
        {"name": "surrogate_rings_1m", "kind": "surrogate", "layout": "leapfrog", "n": 1000000, "precision": "fp32c"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step64", "batch", "rotor", "solve", "solve64", "highorder", "diagnose",
                       "probe", "field", "surrogate"])
    if kind in ("step", "step64"):
        n = _log(rng, 400, 30000 if kind == "step" else 8000)
        return {"kind": "step", "layout": rng.choice(["stations", "gauss"]), "n": n,
                "precision": "fp32c" if kind == "step" else "fp64", "scheme": rng.choice(["rk4", "rk3", "euler"]),
                "steps": rng.choice([1, 1, 2, 10])}
    if kind == "batch":
        return {"kind": "step", "layout": "uneven", "count": rng.randint(2, 24), "nmin": _log(rng, 500, 3000),
                "nmax": _log(rng, 4000, 50000), "precision": "fp32c", "scheme": rng.choice(["rk4", "rk3"]), "steps": 1}
    if kind == "rotor":
        return {"kind": "step", "layout": "rotor", "per_blade": rng.randint(40, 220), "sheds": rng.randint(5, 45),
                "precision": "fp32c", "scheme": rng.choice(["rk3", "rk4"]), "steps": 1, "split": rng.random() < 0.7,
                "inflow": True}
    if kind == "solve":
        return {"kind": "solve", "layout": "gauss", "n": _log(rng, 10000, 400000), "precision": "fp32c",
                "kernel": "gaussian"}
    if kind == "solve64":
        return {"kind": "solve", "layout": rng.choice(["gauss", "stations"]), "n": _log(rng, 2000, 100000),
                "precision": "fp64", "kernel": "gaussian"}
    if kind == "highorder":
        p = rng.choice(["fp32c", "fp32c", "fp64"])
        return {"kind": "solve", "layout": rng.choice(["gauss", "stations"]),
                "n": _log(rng, 1000, 150000 if p == "fp32c" else 40000), "precision": p, "kernel": "highorder"}
    if kind == "diagnose":
        p = rng.choice(["fp32c", "fp32c", "fp64"])
        return {"kind": "diagnose", "layout": rng.choice(["gauss", "stations"]),
                "n": _log(rng, 1000, 150000 if p == "fp32c" else 60000), "precision": p,
                "kernel": rng.choice(["gaussian", "gaussian", "highorder"])}
    if kind == "probe":
        return {"kind": "probe", "layout": rng.choice(["gauss", "stations"]), "n": _log(rng, 1000, 200000),
                "points": _log(rng, 1, 4000), "precision": rng.choice(["fp32c", "fp64"]),
                "kernel": rng.choice(["gaussian", "gaussian", "highorder"])}
    if kind == "field":
        return {"kind": "field", "layout": rng.choice(["gauss", "stations"]), "n": _log(rng, 500, 60000),
                "precision": rng.choice(["fp32c", "fp64"]), "kernel": rng.choice(["gaussian", "gaussian", "highorder"])}
    return {"kind": "surrogate", "layout": rng.choice(["leapfrog", "gauss"]), "n": _log(rng, 60000, 1000000),
            "precision": "fp32c"}


# ---------------------------------------------------------------- inputs
def _wakes(case, seed):
    """The host wakes of a case (one per system)."""
    lay = case["layout"]
    if lay == "uneven":  # the sizes belong to the case, the disturbance of the rings to the seed
        wakes = layouts.uneven_rings(case["count"], case["nmin"], case["nmax"])
        rng = np.random.default_rng(seed)
        for w in wakes:
            w.pos += rng.normal(0.0, 1e-3, w.pos.shape)
        return wakes
    if lay == "rotor":
        s = layouts.RotorShedder(per_blade=case["per_blade"], omega=10.0)
        parts = [s.shed() for _ in range(case["sheds"])]
        rng = np.random.default_rng(seed)
        for age, w in enumerate(reversed(parts)):  # carried down with the inflow since it was shed, and disturbed
            w.pos += age * s.dt * np.array(s.inflow) + rng.normal(0.0, 1e-3, w.pos.shape)
        return [layouts.Wake.concat(parts)]
    n = case["n"]
    if lay == "stations":
        return [layouts.ring_stations(stations=max(8, -(-n // 25)), seed=seed).subset(n)]
    if lay == "leapfrog":
        return [layouts.leapfrog_rings(n, seed=seed)]
    per = 1000 if n >= 150000 else 250 if n >= 10000 else 50
    return [layouts.ring_gaussian(stations=-(-n // per), per_section=per, seed=seed).subset(n)]


def _dt(case):
    return layouts.RotorShedder(omega=10.0).dt if case["layout"] == "rotor" else 0.005


def _points(case, seed):
    """Probe points in and around the ring's core."""
    rng = np.random.default_rng(seed + 7)
    psi = rng.uniform(0.0, 2.0 * math.pi, case["points"])
    rad = 1.0 + rng.normal(0.0, 0.2, case["points"])
    return np.stack([rad * np.cos(psi), rad * np.sin(psi), rng.normal(0.0, 0.2, case["points"])], -1)


def _f64(case):
    return case["precision"] == "fp64" or case["kind"] in ("probe", "field")


def prepare(case, seed):
    wakes = _wakes(case, seed)
    inflow = layouts.RotorShedder().inflow if case.get("inflow") else (0.0, 0.0, 0.0)
    ctx = capi.Context(precision=capi.FP64 if case["precision"] == "fp64" else capi.FP32C, nu=NU, vinf=inflow,
                       kernel=case.get("kernel", "gaussian"), split_positions=bool(case.get("split")))
    ids = [ctx.add_wake(w.n, system=s) for s, w in enumerate(wakes)]
    for k, w in zip(ids, wakes):
        ctx.set_particles(k, w)
    state = {"case": case, "ctx": ctx, "ids": ids, "wakes": wakes}
    if case["kind"] == "probe":
        state["points"] = _points(case, seed)
    if case["kind"] == "surrogate":
        ctx.surrogate_enable(0)
    return state


# ---------------------------------------------------------------- one pass
def run(state):
    case, ctx = state["case"], state["ctx"]
    dtype = np.float64 if _f64(case) else np.float32
    if case["kind"] == "step":
        for k, w in zip(state["ids"], state["wakes"]):
            ctx.set_particles(k, w)
        ctx.step(case["scheme"], _dt(case), case["steps"])
        ctx.sync()
        out = [ctx.state(k) for k in state["ids"]]
        return {"pos": np.concatenate([x for x, _ in out]).astype(dtype, copy=False),
                "alpha": np.concatenate([a for _, a in out]).astype(dtype, copy=False)}
    if case["kind"] in ("solve", "surrogate"):
        ctx.solve()
        v, a = ctx.rates(state["ids"][0])
        return {"velocity": v.astype(dtype, copy=False), "dalpha": a.astype(dtype, copy=False)}
    if case["kind"] == "diagnose":
        record, vbi = ctx.diagnose()
        return {"record": record.astype(dtype, copy=False), "vbi": vbi.astype(dtype, copy=False)}
    if case["kind"] == "probe":
        return {"velocity": ctx.probe(state["points"])}
    return {"field": ctx.vorticity_field(state["ids"][0])}


# ---------------------------------------------------------------- what a pass cannot do without
def _sizes(case):
    if case["layout"] == "uneven":
        return [w.n for w in _wakes(case, 0)]
    if case["layout"] == "rotor":
        return [4 * case["per_blade"] * case["sheds"]]
    return [_wakes(case, 0)[0].n if case["layout"] == "leapfrog" else case["n"]]


def work(case):
    """Bytes: every input and output array once, in FP64.  Flops: per ordered pair, + - x / sqrt counted as one, the
    terms of a pair beyond the reach of the regularisation (59; 95 in full) for the rates, 85 per unordered pair for the
    diagnostics, 30 per probe pair, 20 for the vorticity field, and for the octree the far-field terms of about 2000
    near particles and 1000 cells per target."""
    sizes = _sizes(case)
    n, pairs = sum(sizes), float(sum(m * m for m in sizes))
    kind = case["kind"]
    stages = {"rk4": 4, "rk3": 3, "euler": 1}.get(case.get("scheme"), 1)
    if kind == "step":
        return {"bytes": (8 + 6) * 8.0 * n, "flops": 59.0 * pairs * stages * case["steps"]}
    if kind == "solve":
        return {"bytes": (8 + 6) * 8.0 * n, "flops": (95.0 if case["kernel"] == "highorder" else 59.0) * pairs}
    if kind == "diagnose":
        return {"bytes": 8 * 8.0 * n, "flops": 42.5 * pairs}
    if kind == "probe":
        return {"bytes": 7 * 8.0 * n + 48.0 * case["points"], "flops": 30.0 * n * case["points"]}
    if kind == "field":
        return {"bytes": (7 + 3) * 8.0 * n, "flops": 20.0 * pairs}
    return {"bytes": (8 + 6) * 8.0 * n, "flops": 59.0 * 2000.0 * n + 300.0 * 1000.0 * n}


# ---------------------------------------------------------------- the same in 64 bits
def _cross(a, b):
    return torch.linalg.cross(a, b)


def _gauss_terms(r2, s2):
    """q, F and zeta of the Gaussian kernel; below u = 0.05, where q and F cancel, their Taylor series."""
    u = r2 / s2
    s = s2.sqrt()
    zeta = torch.exp(-0.5 * u) / ((2 * math.pi) ** 1.5 * s ** 3)
    small = u < 0.05
    us = torch.where(small, torch.ones_like(u), u)
    rs = torch.where(small, s2, r2)
    q = (torch.erf((0.5 * us).sqrt()) / (4 * math.pi * s ** 3 * us.sqrt()) - zeta) / us
    f = (zeta - 3 * q) / rs
    ss, tt, term = torch.zeros_like(u), torch.zeros_like(u), torch.ones_like(u)
    for k in range(10):
        ss = ss + term / (2 * k + 3)
        tt = tt + term / (2 * k + 5)
        term = term * (-0.5 * u) / (k + 1)
    c = 1.0 / ((2 * math.pi) ** 1.5 * s ** 3)
    return torch.where(small, c * ss, q), torch.where(small, -c * tt / s2, f), zeta


def _highorder_terms(r2, s2):
    """q, F and the diffusion kernel eta of the high-order algebraic kernel."""
    R = r2 + s2
    q = (r2 + 2.5 * s2) / (4 * math.pi * R ** 2.5)
    f = -3.0 * (r2 + 3.5 * s2) / (4 * math.pi * R ** 3.5)
    return q, f, 13.125 / math.pi * s2 ** 3 / R ** 4.5


def _blocks(n):
    rows = max(1, min(n, 2048))
    return [(t, min(t + rows, n)) for t in range(0, n, rows)], [(s, min(s + 4096, n)) for s in range(0, n, 4096)]


def _exact_rates(x, a, sigma, vol, highorder):
    n = x.shape[0]
    vel, da = torch.zeros_like(x), torch.zeros_like(x)
    hs = 0.5 * sigma ** 2
    tb, sb = _blocks(n)
    for t0, t1 in tb:
        xt, at = x[t0:t1], a[t0:t1]
        sq, sa, sf, sz = (torch.zeros_like(xt) for _ in range(4))
        sw = torch.zeros_like(xt[:, 0])
        for s0, s1 in sb:
            xs, as_ = x[s0:s1], a[s0:s1]
            d = [xt[:, None, m] - xs[None, :, m] for m in range(3)]
            r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
            s2 = hs[t0:t1, None] + hs[None, s0:s1]
            q, f, z = (_highorder_terms if highorder else _gauss_terms)(r2, s2)
            live = (r2 > 0).to(q.dtype)
            q, z = q * live, z * live / s2
            qd = [q * m for m in d]
            p = [m @ as_ for m in qd]  # p[m][:, k] = sum q d_m alpha_k
            sq += torch.stack([p[2][:, 1] - p[1][:, 2], p[0][:, 2] - p[2][:, 0], p[1][:, 0] - p[0][:, 1]], -1)
            sa += q @ as_
            # d . (alpha_t x alpha_s) = alpha_s . (d x alpha_t)
            dot = (d[1] * at[:, None, 2] - d[2] * at[:, None, 1]) * as_[None, :, 0]
            dot += (d[2] * at[:, None, 0] - d[0] * at[:, None, 2]) * as_[None, :, 1]
            dot += (d[0] * at[:, None, 1] - d[1] * at[:, None, 0]) * as_[None, :, 2]
            dot *= f
            sf += torch.stack([(dot * m).sum(1) for m in d], -1)
            sz += z @ as_
            sw += z @ vol[s0:s1]
        vel[t0:t1] = sq
        da[t0:t1] = _cross(at, sa) + sf + 2 * NU * (vol[t0:t1, None] * sz - sw[:, None] * at)
    return vel, da


def _exact_step(case, x, a, sigma, vol, vinf):
    dt = _dt(case)

    def rates(y):
        return torch.cat(_exact_rates(y[:, :3].contiguous(), y[:, 3:].contiguous(), sigma, vol, False), 1)

    y = torch.cat([x, a], 1)
    for _ in range(case["steps"]):
        k1 = rates(y)
        if case["scheme"] == "rk4":
            k2 = rates(y + 0.5 * dt * k1)
            k3 = rates(y + 0.5 * dt * k2)
            k4 = rates(y + dt * k3)
            y = y + dt / 6 * (k1 + 2 * k2 + 2 * k3 + k4)
        elif case["scheme"] == "rk3":
            k2 = rates(y + 0.5 * dt * k1)
            k3 = rates(y + dt * (2 * k2 - k1))
            y = y + dt / 6 * (k1 + 4 * k2 + k3)
        else:
            y = y + dt * k1
        y[:, :3] += dt * vinf
    return y[:, :3], y[:, 3:]


def _exact_diagnose(x, a, sigma, highorder):
    n = x.shape[0]
    hs = 0.5 * sigma ** 2
    hel = ke = kef = en = enf = 0.0
    tb, sb = _blocks(n)
    for t0, t1 in tb:
        xt, at = x[t0:t1], a[t0:t1]
        for s0, s1 in sb:
            xs, as_ = x[s0:s1], a[s0:s1]
            d = [xt[:, None, m] - xs[None, :, m] for m in range(3)]
            r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
            s2 = hs[t0:t1, None] + hs[None, s0:s1]
            # every pair but a particle with itself
            live = torch.arange(t0, t1, device=x.device)[:, None] != torch.arange(s0, s1, device=x.device)[None, :]
            live = live.to(r2.dtype)
            q = (_highorder_terms if highorder else _gauss_terms)(r2, s2)[0] * live
            dot = (d[1] * at[:, None, 2] - d[2] * at[:, None, 1]) * as_[None, :, 0]
            dot += (d[2] * at[:, None, 0] - d[0] * at[:, None, 2]) * as_[None, :, 1]
            dot += (d[0] * at[:, None, 1] - d[1] * at[:, None, 0]) * as_[None, :, 2]
            hel = hel - (q * dot).sum()
            aa = at @ as_.T
            da = (d[0] * at[:, None, 0] + d[1] * at[:, None, 1] + d[2] * at[:, None, 2])
            da = da * (d[0] * as_[None, :, 0] + d[1] * as_[None, :, 1] + d[2] * as_[None, :, 2])
            R = r2 + s2
            w = live / R ** 1.5
            ke = ke + (((r2 + 2 * s2) * aa + da) * w).sum() / (16 * math.pi)
            kef = kef + ((r2 + 1.5 * s2) * aa * w).sum() / (8 * math.pi)
            if highorder:
                w = live / (8 * math.pi * R ** 3.5)
                f1 = 2 * r2 * r2 + 7 * r2 * s2 + 20 * s2 * s2
                f2 = 6 * r2 * r2 + 27 * r2 * s2 + 21 * s2 * s2
                en = en + ((f1 * aa - f2 * da / R) * w).sum()
                enf = enf + (15 * s2 * s2 * aa * w).sum()
    a2 = (a * a).sum(1)
    ke = ke + (a2 / (8 * math.pi * sigma)).sum()
    kef = kef + (3 * a2 / (16 * math.pi * sigma)).sum()
    if highorder:
        en = en + (5 * a2 / (2 * math.pi * sigma ** 3)).sum()
        enf = enf + (15 * a2 / (8 * math.pi * sigma ** 3)).sum()
    xa = _cross(x, a)
    om, rr = a2.sqrt(), x[:, 0] ** 2 + x[:, 1] ** 2
    zc = (om * x[:, 2] * rr).sum() / (om * rr).sum()
    record = [*a.sum(0), *(0.5 * xa.sum(0)), *(_cross(x, xa).sum(0) / 3.0), hel, en, enf, ke, kef, zc]
    q = (_highorder_terms if highorder else _gauss_terms)((x * x).sum(1), sigma ** 2)[0]
    return torch.tensor([float(v) for v in record], dtype=torch.float64), (q[:, None] * _cross(a, -x)).sum(0)


def _exact_probe(pts, x, a, sigma, highorder):
    out = torch.zeros_like(pts)
    for p0 in range(0, pts.shape[0], 512):
        for s0 in range(0, x.shape[0], 16384):
            xs, as_, s2 = x[s0:s0 + 16384], a[s0:s0 + 16384], sigma[s0:s0 + 16384] ** 2
            d = pts[p0:p0 + 512, None, :] - xs[None]
            r2 = (d * d).sum(-1)
            q = (_highorder_terms if highorder else _gauss_terms)(r2, s2[None, :].expand_as(r2))[0]
            out[p0:p0 + 512] += (q[:, :, None] * _cross(as_[None].expand_as(d), d)).sum(1)
    return out


def _exact_field(x, a, sigma, highorder):
    out = torch.zeros_like(x)
    hs = 0.5 * sigma ** 2
    tb, sb = _blocks(x.shape[0])
    for t0, t1 in tb:
        for s0, s1 in sb:
            r2 = ((x[t0:t1, None, :] - x[None, s0:s1, :]) ** 2).sum(-1)
            s2 = hs[t0:t1, None] + hs[None, s0:s1]
            if highorder:
                z = 1.875 / math.pi * s2 ** 2 / (r2 + s2) ** 3.5
            else:
                z = torch.exp(-0.5 * r2 / s2) / ((2 * math.pi) ** 1.5 * s2 ** 1.5)
            out[t0:t1] += z @ a[s0:s1]
    return out


def exact(case, seed):
    wakes = _wakes(case, seed)
    pairs = float(sum(w.n * w.n for w in wakes))
    if case["kind"] == "step":
        pairs *= {"rk4": 4, "rk3": 3, "euler": 1}[case["scheme"]] * case["steps"]
    if case["kind"] == "probe":
        pairs = 4.0 * wakes[0].n * case["points"]
    if pairs > EXACT_PAIRS:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    arrays = [[torch.from_numpy(np.ascontiguousarray(v)).to(dev) for v in (w.pos, w.alpha, w.sigma, w.vol)]
              for w in wakes]
    highorder = case.get("kernel") == "highorder"
    if case["kind"] == "step":
        vinf = layouts.RotorShedder().inflow if case.get("inflow") else (0.0, 0.0, 0.0)
        vinf = torch.tensor(vinf, dtype=torch.float64, device=dev)
        out = [_exact_step(case, *w, vinf) for w in arrays]
        return {"pos": torch.cat([x for x, _ in out]), "alpha": torch.cat([a for _, a in out])}
    x, a, sigma, vol = arrays[0]
    if case["kind"] in ("solve", "surrogate"):
        vel, da = _exact_rates(x, a, sigma, vol, highorder)
        return {"velocity": vel, "dalpha": da}
    if case["kind"] == "diagnose":
        record, vbi = _exact_diagnose(x, a, sigma, highorder)
        return {"record": record, "vbi": vbi}
    if case["kind"] == "probe":
        pts = torch.from_numpy(_points(case, seed)).to(dev)
        return {"velocity": _exact_probe(pts, x, a, sigma, highorder)}
    return {"field": _exact_field(x, a, sigma, highorder)}
