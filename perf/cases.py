"""Timed cases of the engine: what a user's program has it do, through the public Python binding.

Systems come from ``solaris_gb300.scenarios`` (the shapes of the configured
workloads); a case names the shape, its size, the precision of the pair forces
and how many driver calls a pass makes.  ``exact`` restates the model in plain
64-bit torch: GravityAC with its indirect term, Stokes gas drag, RK4, RKF78
with its step control (also for a batch of systems), the integrals, and the
gradient of fixed-step RKF78 through torch's own autograd.
"""
import math

import numpy as np
import torch

from solaris_gb300 import abi, adjoint, engine, scenarios

G = 2.959122082855911025e-4
DEV = "cuda" if torch.cuda.is_available() else "cpu"
PREC = {"fp64": abi.PRECISION_FP64, "split_ff": abi.PRECISION_SPLIT_FF}


def listed():
    return [
        # one Acceleration::Compute call of a small program: a star, two giants, test particles (call latency)
        {"name": "accel_planets_256", "kind": "accel", "shape": "planets", "n": 256, "prec": "fp64"},
        # one evaluation of a self-gravitating disk in the default (reference) arithmetic: ordinary and large
        {"name": "accel_disk_2049", "kind": "accel", "shape": "disk", "n": 2049, "prec": "fp64"},
        {"name": "accel_disk_16411", "kind": "accel", "shape": "disk", "n": 16411, "prec": "fp64"},
        # the same in the split-precision form, a medium odd size
        {"name": "accel_disk_10007_ff", "kind": "accel", "shape": "disk", "n": 10007, "prec": "split_ff"},
        # one RK4 step of the large split-precision disk, host state in and out
        {"name": "rk4_disk_65536_ff", "kind": "rk4", "n": 65536, "prec": "split_ff", "calls": 1},
        # adaptive RKF78 over a planetary system with test particles (the classic small run)
        {"name": "rkf78_planets_256", "kind": "rkf78", "shape": "planets", "n": 256, "calls": 40},
        # the start of a planetesimal run in a gas nebula: drag on 8,190 bodies
        {"name": "rkf78_gas_8193", "kind": "rkf78", "shape": "gas", "n": 8193, "calls": 4},
        # adaptive RKF78 of a small self-gravitating disk
        {"name": "rkf78_disk_1033", "kind": "rkf78", "shape": "disk", "n": 1033, "calls": 2},
        # batched ensembles of uneven systems: initial states in, adaptive RKF78 calls, final states out
        {"name": "ensemble_512", "kind": "ensemble", "systems": 512, "prec": "fp64", "calls": 4},
        {"name": "ensemble_1024_ff", "kind": "ensemble", "systems": 1024, "prec": "split_ff", "calls": 4},
        # gradient of a final-state misfit through fixed-step RKF78 (forward and backward)
        {"name": "adjoint_1033", "kind": "adjoint", "n": 1033, "steps": 8, "every": 4},
        # energy, momentum and barycentre of a large system, as an output record needs them
        {"name": "integrals_24000", "kind": "integrals", "n": 24000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["accel", "accel", "accel", "rk4", "rkf78", "rkf78", "ensemble", "adjoint", "integrals"])
    if kind == "accel":
        shape, prec = rng.choice([("planets", "fp64"), ("disk", "fp64"), ("disk", "split_ff")])
        n = _log(rng, 40, 8000) if shape == "planets" else _log(rng, 257, 20011) if prec == "fp64" else _log(rng, 1025, 65536)
        return {"kind": kind, "shape": shape, "n": n, "prec": prec}
    if kind == "rk4":
        return {"kind": kind, "n": _log(rng, 4096, 65536), "prec": "split_ff", "calls": 1}
    if kind == "rkf78":
        shape = rng.choice(["planets", "gas", "disk"])
        if shape == "planets":
            return {"kind": kind, "shape": shape, "n": _log(rng, 30, 2000), "calls": rng.randint(5, 40)}
        if shape == "gas":
            return {"kind": kind, "shape": shape, "n": _log(rng, 300, 8193), "calls": 4}
        return {"kind": kind, "shape": shape, "n": _log(rng, 265, 2100), "calls": rng.randint(1, 3)}
    if kind == "ensemble":
        return {"kind": kind, "systems": _log(rng, 32, 1024), "prec": rng.choice(["fp64", "split_ff"]), "calls": rng.randint(2, 4)}
    if kind == "adjoint":
        return {"kind": kind, "n": _log(rng, 129, 1500), "steps": rng.randint(3, 8), "every": rng.randint(2, 5)}
    return {"kind": kind, "n": _log(rng, 1025, 60000)}


# ---- inputs ----------------------------------------------------------------------
def _system(case, seed):
    n, kind = case["n"], case["kind"]
    shape = {"adjoint": "embryos", "rk4": "disk", "integrals": "disk"}.get(kind) or case["shape"]
    if shape == "planets":
        return scenarios.config1(seed=seed, n_tp=n - 3)
    if shape == "gas":
        return scenarios.config2(seed=seed, n_pl=n - 3)
    if shape == "embryos":
        return scenarios.config5(seed=seed, n_pl=n - 9)
    return scenarios.config3(seed=seed, n=n)


def _first_step(case, s):
    """The trial step of the first driver call: near the natural step, or the
    simulator's own start (shortest period / 50,000) for the run in gas."""
    if case["kind"] == "rk4" or case["kind"] == "adjoint":
        return 100.0 * s.h0
    return {"planets": 250.0, "gas": 1.0, "disk": 300.0}[case["shape"]] * s.h0


def _ensemble(case, seed):
    """Systems of a star, 2 to 12 planets and up to 512 test particles (the
    distributions of scenarios.config4): their sizes belong to the case, the
    orbits to the seed."""
    sizes, rng = np.random.default_rng(case["systems"]), np.random.default_rng(seed)
    systems, hs = [], []
    for _ in range(case["systems"]):
        npl, ntp = int(sizes.integers(2, 13)), int(sizes.integers(0, 513))
        k = npl + ntp
        m = np.exp(rng.uniform(math.log(1e-6), math.log(1e-3), npl))
        a = np.exp(rng.uniform(math.log(0.1), math.log(30.0), k))
        mu = abi.GAUSS2 * (1.0 + np.concatenate([m, np.zeros(ntp)]))
        ph = scenarios.elements_to_phase(mu, a, rng.uniform(0.0, 0.2, k), np.zeros(k), *rng.uniform(0.0, 2.0 * np.pi, (3, k)))
        star = (abi.CENTRAL_BODY, {"mass": [1.0], "phase": np.zeros((1, 6))})
        groups = [star, (abi.GIANT_PLANET, {"mass": m, "phase": ph[:npl]}),
                  (abi.TEST_PARTICLE, {"mass": np.zeros(ntp), "phase": ph[npl:]})]
        systems.append(scenarios._assemble("member", groups, epsilon=1.0e-10))
        hs.append(scenarios.orbital_period(abi.GAUSS2, float(a.min())) / 50.0)
    return systems, [s.y0 for s in systems], [0.0] * len(systems), hs


def prepare(case, seed):
    if case["kind"] == "ensemble":
        systems, y0s, times, hs = _ensemble(case, seed)
        return {"case": case, "ens": engine.Ensemble(systems, precision=PREC[case["prec"]]), "y0s": y0s, "times": times, "hs": hs}
    s = _system(case, seed)
    st = {"case": case, "s": s, "ctx": engine.Context(s, precision=PREC[case.get("prec", "fp64")])}
    if case["kind"] in ("rk4", "rkf78"):
        st["h"] = _first_step(case, s)
    if case["kind"] == "adjoint":
        st["h"] = _first_step(case, s)
        st["grad"] = torch.from_numpy(_misfit_gradient(s, seed))
    return st


def _misfit_gradient(s, seed):
    """d/dy of a squared final-position misfit against some target: position rows only."""
    g = np.zeros((s.n, 6))
    g[1:, :3] = 2.0 * np.random.default_rng(seed + 17).normal(0.0, 1.0e-3, (s.n - 1, 3))
    return g.ravel()


# ---- one pass ----------------------------------------------------------------------
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "ensemble":
        ens = st["ens"]
        ens.set_state(st["y0s"], st["times"], st["hs"])
        stats = ens.advance(case["calls"])
        ys, lines, status = ens.get_state()
        return {"y": np.concatenate(ys), "lines": np.asarray(lines), "status": status, "stats": list(stats)}
    s, ctx = st["s"], st["ctx"]
    if kind == "accel":
        dydt, rm3, nn, nd = ctx.accel(0.0, s.y0)
        return {"dydt": dydt, "rm3": rm3, "nn": nn, "nd": nd}
    if kind == "integrals":
        return {"out": ctx.integrals(s.y0)}
    if kind == "adjoint":
        y0 = torch.from_numpy(s.y0).requires_grad_(True)
        mass = torch.from_numpy(s.mass).requires_grad_(True)
        y = adjoint.integrate(ctx, y0, mass, st["h"], case["steps"], case["every"])
        dy0, dmass = torch.autograd.grad(y, (y0, mass), st["grad"])
        return {"y": y.detach(), "dy0": dy0, "dmass": dmass}
    ctx.set_state(s.y0)
    r = ctx.driver(abi.RUNGE_KUTTA4 if kind == "rk4" else abi.RUNGE_KUTTA_FEHLBERG78, 0.0, st["h"], case["calls"])
    return {"y": ctx.get_state(), "time": r["time"], "h_next": r["h_next"], "h_did": r["h_did"], "stats": list(r["stats"])}


# ---- what a pass cannot do without ------------------------------------------------------
def _pairs(case):
    """Pair terms of one evaluation: the Kepler terms and the direct terms of GravityAC."""
    n = case["n"]
    shape = {"adjoint": "embryos", "rk4": "disk"}.get(case["kind"]) or case["shape"]
    return n * 3 if shape in ("planets", "gas") else (n - 1) * (n - 1)


def work(case):
    kind = case["kind"]
    if kind == "ensemble":  # 272 bodies and 6 attracting planets a system on average, 13 evaluations a call
        s, k = case["systems"], case["calls"]
        return {"bytes": 2.0 * 8 * 6 * 272 * s, "flops": 1.0 * s * k * 272 * (13 * 7 * 20 + 6 * 140)}
    n = case["n"]
    if kind == "accel":
        return {"bytes": 8.0 * 6 * n * 2 + 20.0 * n, "flops": 20.0 * _pairs(case)}
    if kind == "integrals":
        return {"bytes": 8.0 * 7 * n, "flops": 10.0 * n * (n - 1) / 2}
    if kind == "rk4":
        return {"bytes": 8.0 * 6 * n * 2, "flops": case["calls"] * (4 * 20.0 * _pairs(case) + 6 * n * 14)}
    if kind == "rkf78":
        drag = 60.0 * n if case["shape"] == "gas" else 0.0
        return {"bytes": 8.0 * 6 * n * 2, "flops": case["calls"] * (13 * (20.0 * _pairs(case) + drag) + 6.0 * n * 140)}
    # adjoint: 11 evaluations forward and 11 transposed Jacobians (twice a pair's work) a step
    return {"bytes": 8.0 * 6 * n * 4, "flops": case["steps"] * (11 * (20.0 + 40.0) * _pairs(case) + 6.0 * n * 200)}


# ---- the same results in plain 64-bit torch -----------------------------------------------
def _t(a):
    return torch.as_tensor(np.asarray(a, np.float64), device=DEV)


class _Model:
    """dy/dt of a batch of systems: y (S, n, 6); mass (S, n); the first `few`
    bodies of a system attract every body, the rest nothing."""

    def __init__(self, mass, few, live, drag=None):
        self.m, self.few, self.live, self.drag = mass, few, live, drag

    def __call__(self, y):
        r = y[..., :3]
        m = self.m
        d2 = (r * r).sum(-1)
        rm3 = torch.where(d2 > 0, d2, torch.ones_like(d2)) ** -1.5 * (d2 > 0)
        a = -G * (m[..., :1] + m)[..., None] * r * rm3[..., None]
        k = self.few
        gm = (G * m[..., :k]).clone()
        gm[..., 0] = 0.0
        src, ind = r[..., :k, :], (r * rm3[..., None])[..., :k, :]
        parts = []
        step = max(1, (1 << 25) // max(1, k * r.shape[0]))
        for lo in range(0, r.shape[-2], step):
            d = src[..., None, :, :] - r[..., lo:lo + step, None, :]
            q = (d * d).sum(-1)
            near = q > 0
            w = torch.where(near, q, torch.ones_like(q)) ** -1.5 * near * gm[..., None, :]
            direct = (w[..., None] * d).sum(-2)
            # a body has no indirect term of its own: only of the others
            own = torch.zeros_like(direct)
            if lo < k:
                hi = min(k, lo + step)
                own[..., :hi - lo, :] = gm[..., lo:hi, None] * ind[..., lo:hi, :]
            parts.append(direct - ((gm[..., None] * ind).sum(-2)[..., None, :] - own))
        a = a + torch.cat(parts, -2)
        if self.drag is not None:
            a = a + self.drag(y)
        mask = self.live.clone()
        mask[..., 0] = 0.0
        return torch.cat([y[..., 3:], a], -1) * mask[..., None]


def _stokes_drag(s):
    g = s.gas
    gs, radius = _t(s.gamma_stokes)[None], _t(s.radius)[None]
    small = torch.as_tensor(np.asarray(s.type) == abi.PLANETESIMAL, device=DEV)[None]

    def drag(y):
        x, yy, z = y[..., 0], y[..., 1], y[..., 2]
        r = (x * x + yy * yy + z * z).sqrt()
        rc = (x * x + yy * yy).sqrt()
        safe = torch.where(small, rc, torch.ones_like(rc))
        assert bool((radius[small] >= 10.0 * g["mean_free_path"][0] * r[small] ** g["mean_free_path"][1]).all())
        vc = (G * float(s.mass[0]) / safe).sqrt() * (1.0 - 2.0 * g["eta"][0] * safe ** g["eta"][1]).sqrt()
        u = torch.stack([y[..., 3] + vc * yy / safe, y[..., 4] - vc * x / safe, y[..., 5]], -1)
        h = g["scale_height"][0] * safe ** g["scale_height"][1]
        rho = g["density"][0] * safe ** g["density"][1] * torch.exp(-(z / h) ** 2)
        c = gs * u.norm(dim=-1) * rho
        return torch.where(small[..., None], -c[..., None] * u, torch.zeros_like(u))

    return drag


def _model(s):
    c = s.counts
    few = c[0] + c[1] + c[2] + c[3] + c[4]
    return _Model(_t(s.mass)[None], few, torch.ones(1, s.n, dtype=torch.float64, device=DEV), _stokes_drag(s) if s.gas else None)


_A = [[], [2 / 27], [1 / 36, 1 / 12], [1 / 24, 0, 1 / 8], [5 / 12, 0, -25 / 16, 25 / 16], [1 / 20, 0, 0, 1 / 4, 1 / 5],
      [-25 / 108, 0, 0, 125 / 108, -65 / 27, 125 / 54], [31 / 300, 0, 0, 0, 61 / 225, -2 / 9, 13 / 900],
      [2, 0, 0, -53 / 6, 704 / 45, -107 / 9, 67 / 90, 3],
      [-91 / 108, 0, 0, 23 / 108, -976 / 135, 311 / 54, -19 / 60, 17 / 6, -1 / 12],
      [2383 / 4100, 0, 0, -341 / 164, 4496 / 1025, -301 / 82, 2133 / 4100, 45 / 82, 45 / 164, 18 / 41],
      [3 / 205, 0, 0, 0, 0, -6 / 41, -3 / 205, -3 / 41, 3 / 41, 6 / 41, 0],
      [-1777 / 4100, 0, 0, -341 / 164, 4496 / 1025, -289 / 82, 2193 / 4100, 51 / 82, 33 / 164, 12 / 41, 0, 1]]
_B = [41 / 840, 0, 0, 0, 0, 34 / 105, 9 / 35, 9 / 35, 9 / 280, 9 / 280, 41 / 840]


def _sum(coefs, f):
    acc = None
    for c, v in zip(coefs, f):
        if c:
            acc = c * v if acc is None else acc + c * v
    return acc


def _stages(model, y, f0, h, last):
    f = [f0]
    for r in range(1, last + 1):
        f.append(model(y + h * _sum(_A[r], f)))
    return f


def _rkf78(model, y, h, eps, calls):
    """RKF78 driver calls of a batch, each system with its own adaptive step."""
    S = y.shape[0]
    t, did = torch.zeros_like(h), torch.zeros_like(h)
    acc = rej = 0
    for _ in range(calls):
        f0 = model(y)
        hb = h.clone()
        scale = y.abs() + (hb.view(S, 1, 1) * f0).abs() + 1.0e-30
        open_ = torch.ones(S, dtype=torch.bool, device=y.device)
        out = y
        while bool(open_.any()):
            hv = hb.view(S, 1, 1)
            f = _stages(model, y, f0, hv, 12)
            err = hv * (f[0] + f[10] - f[11] - f[12]).abs() * 41.0 / 840.0
            em = (err / scale).abs().flatten(1).amax(1) / eps
            ok = open_ & (em < 1.0)
            out = torch.where(ok.view(S, 1, 1), y + hv * _sum(_B, f), out)
            t, did = torch.where(ok, t + hb, t), torch.where(ok, hb, did)
            h = torch.where(ok, torch.where(em > 1.89e-4, 0.9 * hb * em ** -0.2, 5.0 * hb), h)
            hb = torch.where(open_ & ~ok, torch.maximum(0.9 * hb * em ** -0.25, 0.1 * hb), hb)
            acc, rej = acc + int(ok.sum()), rej + int((open_ & ~ok).sum())
            open_ = open_ & ~ok
        y = out
    return y, t, h, did, acc, rej


def _back(x):
    return x.detach().reshape(-1).cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    with torch.no_grad():
        if kind == "ensemble":
            return _exact_ensemble(case, seed)
        s = _system(case, seed)
        y = _t(s.y0).reshape(1, s.n, 6)
        if kind == "accel":
            return _exact_accel(s, y)
        if kind == "integrals":
            return {"out": _exact_integrals(s)}
        if kind == "rk4":
            f, h = _model(s), _first_step(case, s)
            for _ in range(case["calls"]):
                k1 = f(y)
                k2 = f(y + h * 0.5 * k1)
                k3 = f(y + h * 0.5 * k2)
                k4 = f(y + h * k3)
                y = y + h * (k1 / 6 + k2 / 3 + k3 / 3 + k4 / 6)
            return {"y": _back(y), "time": h * case["calls"], "h_next": h, "h_did": h, "stats": None}
        if kind == "rkf78":
            y, t, h, did, _, _ = _rkf78(_model(s), y, _t([_first_step(case, s)]), float(s.epsilon), case["calls"])
            return {"y": _back(y), "time": float(t[0]), "h_next": float(h[0]), "h_did": float(did[0]), "stats": None}
    model, h = _model(s), _first_step(case, s)
    y0 = y.clone().requires_grad_(True)
    model.m = model.m.clone().requires_grad_(True)
    z = y0
    for _ in range(case["steps"]):
        z = z + h * _sum(_B, _stages(model, z, model(z), h, 10))
    dy0, dm = torch.autograd.grad(z, (y0, model.m), _t(_misfit_gradient(s, seed)).reshape(1, s.n, 6))
    return {"y": _back(z), "dy0": _back(dy0), "dmass": _back(dm)}


def _exact_accel(s, y):
    f = _model(s)(y)[0]
    r = y[0, :, :3]
    d2 = (r * r).sum(-1)
    rm3 = torch.where(d2 > 0, torch.where(d2 > 0, d2, torch.ones_like(d2)) ** -1.5, torch.zeros_like(d2))
    c = s.counts
    k = c[0] + c[1] + c[2] + c[3] + c[4]
    nd = torch.zeros(s.n, dtype=torch.float64, device=DEV)
    for lo in range(1, s.n, 1024):
        hi = min(s.n, lo + 1024)
        q = ((r[None, 1:k] - r[lo:hi, None]) ** 2).sum(-1)
        rows = torch.arange(lo, hi, device=DEV)
        own = rows < k
        q[(rows - lo)[own], rows[own] - 1] = math.inf
        nd[lo:hi] = q.amin(1).sqrt()
    return {"dydt": _back(f), "rm3": _back(rm3), "nn": None, "nd": _back(nd)}


def _exact_integrals(s):
    y, m = s.y0.reshape(-1, 6), s.mass
    c = s.counts
    M = math.fsum(m[:c[0] + c[1] + c[2] + c[3]])
    bc = [math.fsum(m * y[:, k]) / M for k in range(6)]
    ang = [math.fsum(m * v) for v in np.cross(y[:, :3], y[:, 3:]).T]
    ke = math.fsum(0.5 * m * (y[:, 3:] ** 2).sum(1))
    r, mt, pe = _t(y[:, :3]), _t(m), 0.0
    for lo in range(0, s.n, 1024):
        q = ((r[None] - r[lo:lo + 1024, None]) ** 2).sum(-1)
        w = torch.where(q > 0, q, torch.ones_like(q)) ** -0.5 * (q > 0)
        pe += float((mt[lo:lo + 1024, None] * w * mt[None]).sum())
    pe *= 0.5 * G
    return np.array([M, *bc, math.dist(bc[:3], (0, 0, 0)), math.dist(bc[3:], (0, 0, 0)), *ang, math.dist(ang, (0, 0, 0)), ke, pe, ke - pe])


def _exact_ensemble(case, seed):
    systems, y0s, _, hs = _ensemble(case, seed)
    S, n = len(systems), max(s.n for s in systems)
    y, m, live = np.zeros((S, n, 6)), np.zeros((S, n)), np.zeros((S, n))
    for k, s in enumerate(systems):
        y[k, :s.n], m[k, :s.n], live[k, :s.n] = y0s[k].reshape(-1, 6), s.mass, 1.0
    few = max(s.counts[0] + s.counts[1] for s in systems)
    out, t, h, did, _, _ = _rkf78(_Model(_t(m), few, _t(live)), _t(y), _t(hs), 1.0e-10, case["calls"])
    out = out.cpu().numpy()
    flat = np.concatenate([out[k, :s.n].ravel() for k, s in enumerate(systems)])
    return {"y": flat, "lines": torch.stack([t, h, did], 1).cpu().numpy(), "status": None, "stats": None}
