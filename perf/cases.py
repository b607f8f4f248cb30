"""The workloads this library is timed on, each through its public entry points.

The library keeps one registered case (and one network) per process, as the
reference keeps its module state, so the states of one case share its
registration: the grid, the metrics, the launch shapes and the captured step
are laid out once, and each state brings its own flow field.  A pass of a flow
case is what a program with a restart file does: the freestream start, its own
q (and nu_t) uploaded, the start-up boundary conditions, a number of
iterations with their residual history, and the solution read back.
"""
from __future__ import annotations

import ctypes
import json
import math

import numpy as np
import torch

from aerocfd_b200 import _lib, case as case_mod, grids, solver, warmstart
from aerocfd_b200.case import Config

GAMMA = 1.4


def listed():
    return [
        # the smallest call: a 33 x 17 x 5 Euler channel, where launches and latency count
        {"name": "bump_small", "kind": "bump", "ni": 33, "nj": 17, "nk": 5, "inviscid": 4, "mixed": False,
         "viscous": False, "iters": 50},
        # the Euler bump channel 97 x 49 x 5 with Steger-Warming + WENO5
        {"name": "bump_weno5", "kind": "bump", "ni": 97, "nj": 49, "nk": 5, "inviscid": 5, "mixed": False,
         "viscous": False, "iters": 50},
        # the laminar NACA0012 O-grid, 4 blocks of 129 x 65 x 3, Roe + WENO3
        {"name": "naca_laminar", "kind": "naca", "nblk": 4, "ni": 129, "nj": 65, "nk": 3, "sa": False,
         "inviscid": 4, "mixed": False, "iters": 50},
        # the same section in 2-D mode with the SA model
        {"name": "naca_2d_sa", "kind": "naca", "nblk": 4, "ni": 129, "nj": 65, "nk": 1, "sa": True,
         "inviscid": 4, "mixed": False, "iters": 50},
        # the aerofoil driven call by call, as a Fortran program with its call sites routed here does
        {"name": "naca_dropin", "kind": "dropin", "nblk": 4, "ni": 129, "nj": 65, "nk": 3, "iters": 10},
        # one flux call on arrays that were never registered (a single call site being switched)
        {"name": "flux_transient", "kind": "flux", "ni": 97, "nj": 49, "nk": 5},
        # the turbulent flat plate 193 x 129 x 33 as 8 blocks, SA, tuned once, in FP64 and in mixed precision
        {"name": "plate_sa", "kind": "plate", "nbi": 8, "nbj": 1, "nbk": 1, "ni": 193, "nj": 129, "nk": 33,
         "mixed": False, "tuned": True, "iters": 40},
        {"name": "plate_sa_mixed", "kind": "plate", "nbi": 8, "nbj": 1, "nbk": 1, "ni": 193, "nj": 129, "nk": 33,
         "mixed": True, "tuned": True, "iters": 40},
        # a sweep of 64 uneven bump channels as one batch in mixed precision, tuned once
        {"name": "bump_batch", "kind": "batch", "ncase": 64, "sweep": 0, "mixed": True, "tuned": True, "iters": 40},
        # a family of 8 NACA sections with SA as one batch (the data a warm start is trained on)
        {"name": "naca_family", "kind": "family", "members": 8, "ni": 129, "nj": 65, "nk": 3, "iters": 20},
        # the unsteady dual-time Crank-Nicolson advance of a viscous bump channel
        {"name": "bump_crank", "kind": "crank", "ni": 97, "nj": 49, "nk": 5, "iters": 10},
        # the warm-start network: Adam steps on solver samples, then the prediction of a held-out member
        {"name": "warmstart_mlp", "kind": "mlp", "width": 256, "depth": 8, "batch": 8192, "rows": 131072,
         "predict": 33540, "steps": 40},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["bump", "bump", "naca", "naca", "dropin", "flux", "plate", "plate", "batch", "family", "crank",
                       "mlp"])
    if kind in ("bump", "crank", "flux"):
        c = {"kind": kind, "ni": _log_int(rng, 17, 257), "nj": _log_int(rng, 9, 97), "nk": rng.randint(3, 9)}
        if kind == "bump":
            c.update(inviscid=rng.choice([4, 4, 5, 8]), mixed=rng.random() < 0.4, viscous=rng.random() < 0.4,
                     iters=rng.randint(20, 60))
        if kind == "crank":
            c.update(iters=rng.randint(4, 10))
        return c
    if kind == "naca":
        nk = rng.choice([1, 3, 3, 5])
        return {"kind": kind, "nblk": rng.choice([2, 4]), "ni": 2 * _log_int(rng, 16, 64) + 1,
                "nj": _log_int(rng, 17, 65), "nk": nk, "sa": rng.random() < 0.5, "inviscid": rng.choice([4, 4, 8]),
                "mixed": rng.random() < 0.4, "iters": rng.randint(20, 50)}
    if kind == "dropin":
        return {"kind": kind, "nblk": rng.choice([2, 4]), "ni": 2 * _log_int(rng, 16, 64) + 1,
                "nj": _log_int(rng, 17, 65), "nk": 3, "iters": rng.randint(4, 10)}
    if kind == "plate":
        nbi, nbj, nbk = rng.choice([(8, 1, 1), (4, 1, 1), (2, 1, 1), (6, 1, 1), (2, 2, 2)])
        bi, bj, bk = _log_int(rng, 12, 25), _log_int(rng, 24, 65), rng.randint(4, 17)
        return {"kind": kind, "nbi": nbi, "nbj": nbj, "nbk": nbk, "ni": nbi * (bi - 1) + 1, "nj": nbj * (bj - 1) + 1,
                "nk": nbk * (bk - 1) + 1, "mixed": rng.random() < 0.5, "tuned": rng.random() < 0.5,
                "iters": rng.randint(10, 40)}
    if kind == "batch":
        return {"kind": kind, "ncase": rng.randint(3, 40), "sweep": rng.randint(1, 1000), "mixed": rng.random() < 0.6,
                "tuned": rng.random() < 0.5, "iters": rng.randint(10, 40)}
    if kind == "family":
        return {"kind": kind, "members": rng.randint(2, 6), "ni": 2 * _log_int(rng, 24, 64) + 1,
                "nj": _log_int(rng, 33, 65), "nk": 3, "iters": rng.randint(10, 20)}
    return {"kind": "mlp", "width": rng.choice([128, 256]), "depth": rng.randint(3, 8),
            "batch": 512 * rng.randint(2, 16), "rows": rng.randint(20000, 131072), "predict": rng.randint(1000, 33540),
            "steps": rng.randint(10, 40)}


# ------------------------------------------------------------------ the cases
def _flow_case(c):
    """The case's blocks and, for a batch, each block's own Control.in values."""
    k = c["kind"]
    if k in ("bump", "crank"):
        ns = k == "crank" or c["viscous"]
        cfg = Config(solver=case_mod.IFLAG_NSSOLVER if ns else case_mod.IFLAG_EULERSOLVER, ma=0.5,
                     re=2000.0 if ns else 1.0e6, cfl=3.0 if ns else 5.0, inviscid=c.get("inviscid", 4))
        if k == "crank":
            cfg.time, cfg.timeadvance, cfg.dt = case_mod.IFLAG_UNSTEADY, case_mod.IFLAG_2NDCRANK, 2.0e-3
        return grids.bump_channel(c["ni"], c["nj"], c["nk"], cfg=cfg), None
    if k in ("naca", "dropin"):
        two = c["nk"] == 1
        cfg = Config(solver=case_mod.IFLAG_NSSOLVER, ma=0.5, re=5000.0, aoa_deg=2.0, cfl=2.0,
                     inviscid=c.get("inviscid", 4), dimension=case_mod.IFLAG_2D if two else case_mod.IFLAG_3D)
        if c.get("sa"):
            cfg.turbulence, cfg.re, cfg.nutinf = case_mod.IFLAG_SA, 1.0e5, 3.0
        return grids.naca_ogrid(c["nblk"], c["ni"], c["nj"], c["nk"], cfg=cfg), None
    if k == "plate":
        cfg = Config(solver=case_mod.IFLAG_NSSOLVER, turbulence=case_mod.IFLAG_SA, ma=0.2, re=5.0e6, cfl=5.0,
                     nutinf=3.0)
        return grids.flat_plate(c["nbi"], c["nbj"], c["nbk"], c["ni"], c["nj"], c["nk"], cfg=cfg), None
    if k == "batch":
        return grids.batch_case(grids.bump_batch(c["ncase"], seed=c["sweep"]))
    if k == "family":
        return grids.batch_case([m for m, _ in warmstart.naca_family(c["members"], seed=0, ni=c["ni"], nj=c["nj"],
                                                                     nk=c["nk"])])
    raise ValueError(k)


class Registered:
    """The registered case: its q (and nu_t) arrays lie one after another in one
    buffer, each on its own pages, so a state's field is one copy."""

    def __init__(self, c):
        self.case, params = _flow_case(c)
        blocks = self.case.blocks
        names = ["q"] + (["nut"] if self.case.cfg.turbulence else []) + (["q0"] if c["kind"] == "crank" else [])
        self.names, page, total, spans = names, 512, 0, []
        for n in names:
            for b in blocks:
                spans.append((n, b, total))
                total += -(-b.fields[n].size // page) * page
        self.buf = torch.zeros(total + page, dtype=torch.float64)
        skip = (-self.buf.data_ptr() // 8) % page
        self.buf = self.buf[skip:skip + total]
        flat = self.buf.numpy()
        for n, b, off in spans:
            a = b.fields[n]
            b.fields[n] = flat[off:off + a.size].reshape(a.shape)
        self.spans = spans
        self.gc = solver.GpuCase(self.case, block_params=params)
        self.cfgs = params or {b.m: self.case.cfg for b in blocks}
        self.gc.compute_geometry()
        self.gc.sync_to_host(solver.mask("x", "y", "z"))
        self.gc.init_flowfield()
        self.gc.start()
        self.gc.set_precision(bool(c.get("mixed")))
        if c["kind"] != "dropin":
            self.gc.use_graphs(True)
        if c.get("tuned"):
            self.gc.autotune(2)

    def field(self, seed):
        """A smooth disturbance of the freestream, a function of the coordinates
        alone so that blocks agree at their interfaces."""
        rng = np.random.default_rng(seed)
        waves = [(rng.uniform(-4, 4, 3), rng.uniform(0, 2 * np.pi, 5)) for _ in range(3)]
        out = torch.zeros_like(self.buf)
        flat = out.numpy()
        for n, b, off in self.spans:
            cfg = self.cfgs[b.m]
            X, Y, Z = (np.clip(b.fields[v], -2.0, 3.0) for v in ("x", "y", "z"))
            d = 0.0
            for kv, ph in waves:
                d = d + np.sin((kv[0] * X + kv[1] * Y + kv[2] * Z)[..., None] + ph) * (0.01 / len(waves))
            a = math.radians(cfg.aoa_deg)
            rho, u, v, w = 1.0 + d[..., 0], math.cos(a) * (1.0 + d[..., 1]), math.sin(a) + d[..., 2], 0.0 * d[..., 3]
            p = (1.0 + d[..., 4]) / (GAMMA * cfg.ma ** 2)
            at = flat[off:off + b.fields[n].size].reshape(b.fields[n].shape)
            if n == "nut":
                at[...] = cfg.nutinf * (1.0 + 5.0 * d[..., 3])
                continue
            q = np.stack([rho, rho * u, rho * v, rho * w,
                          p / (GAMMA - 1.0) + 0.5 * rho * (u * u + v * v + w * w)], -1)
            at[...] = q if n == "q" else np.repeat(q, 2, axis=-1)
        return out


_now = {"key": None, "reg": None, "net": None}


def _drop():
    if _now["reg"] is not None:
        _now["reg"].gc.close()
    if _now["net"] is not None:
        _now["net"].close()
    _now.update(key=None, reg=None, net=None)


def _registered(c):
    key = json.dumps({k: v for k, v in c.items() if k != "name"}, sort_keys=True)
    if _now["key"] != key:
        _drop()
        _now["reg"] = Registered(c)
        _now["key"] = key
    return _now["reg"]


def _samples(rng, n):
    """Node features of NACA family members and a smooth field on them."""
    x = np.concatenate([rng.uniform(-1, 1, (n, 2)), rng.uniform(-1.3, 1.3, (n, 1)), rng.uniform(-1, 1, (n, 6))], 1)
    near = np.exp(-2.0 * (x[:, 2:3] + 1.3))
    t = np.concatenate([0.1 * np.sin(2 * x[:, 0:1] + x[:, 3:4]) * near, -near, 0.2 * x[:, 1:2] * near,
                        0.3 * np.cos(3 * x[:, 0:1]) * near * (1 + x[:, 7:8]), 3 * near * x[:, 8:9]], 1)
    return x.astype(np.float32), t.astype(np.float32)


def prepare(case, seed):
    c, rng = case, np.random.default_rng(seed)
    if c["kind"] == "flux":
        return _prepare_flux(c, rng)
    if c["kind"] == "mlp":
        _drop()
        _now["net"] = warmstart.Network(n_in=9, n_out=5, width=c["width"], depth=c["depth"], batch=c["batch"], seed=1)
        x, t = _samples(rng, c["rows"])
        return {"case": c, "x": x, "t": t, "new": _samples(rng, c["predict"])[0]}
    reg = _registered(c)
    return {"case": c, "reg": reg, "field": reg.field(seed)}


def run(state):
    c = state["case"]
    if c["kind"] == "flux":
        return _run_flux(state)
    if c["kind"] == "mlp":
        net = _now["net"]
        loss = net.train(state["x"], state["t"], c["steps"], lr=1.0e-3)
        return {"loss": loss, "predicted": net.predict(state["new"])}
    reg = state["reg"]
    gc, m = reg.gc, solver.mask(*reg.names)
    gc.init_flowfield()
    reg.buf.copy_(state["field"])
    gc.sync_to_device(m)
    gc.start()
    hist = _dropin(reg, c["iters"]) if c["kind"] == "dropin" else gc.step(c["iters"])
    gc.sync_to_host(m)
    return {"solution": reg.buf, "history": hist}


def _dropin(reg, iters):
    """main.f90:343-447 call by call on registered arrays."""
    gc, hist = reg.gc, np.zeros((iters, 7))
    for s in range(iters):
        for b in reg.case.blocks:
            gc.get_primitivevariables(b)
            gc.inviscid_flux_1(b)
            gc.viscous_flux(b)
            gc.find_dt(b)
            gc.implicit1st(b)
        gc.physical_bc()
        gc.updatebuffer()
        gc.average1()
        gc.average2()
        for b in reg.case.blocks:
            gc.get_primitivevariables(b)
        hist[s] = gc.residual()
    return hist


# ------------------------------------------------- one flux call, transient mode
def _flux_arrays(c, rng):
    """q, a curvilinear set of metrics and 1/J on one block, (k, j, i, component)."""
    nk, nj, ni = c["nk"], c["nj"], c["ni"]
    k, j, i = np.meshgrid(np.arange(nk) / nk, np.arange(nj) / nj, np.arange(ni) / ni, indexing="ij")
    ph = rng.uniform(0, 2 * np.pi, 32)
    wave = [np.sin(6 * i + 4 * j + 2 * k + p) for p in ph]
    rho, u, v, w = 1 + 0.1 * wave[0], 1 + 0.1 * wave[1], 0.1 * wave[2], 0.05 * wave[3]
    p = (1 + 0.1 * wave[4]) / (GAMMA * 0.25)
    q = np.stack([rho, rho * u, rho * v, rho * w, p / (GAMMA - 1) + 0.5 * rho * (u * u + v * v + w * w)], -1)
    scale = [ni / 3.0, nj, nk / 0.2]
    dx = np.stack([scale[n // 3] * ((1.0 if n // 3 == n % 3 else 0.0) + 0.05 * wave[5 + n]) for n in range(9)], -1)
    inv_j = (1 + 0.1 * wave[15]) / (scale[0] * scale[1] * scale[2])
    return [np.ascontiguousarray(a) for a in (q, dx, inv_j)]


def _prepare_flux(c, rng):
    q, dx, inv_j = _flux_arrays(c, rng)
    _drop()
    _lib.check(_lib.load().aero_init(0), "aero_init")
    box = [1, c["ni"], 1, c["nj"], 1, c["nk"]]
    ints = (ctypes.c_int * 18)(*(box + box + [2, c["ni"] - 1, 2, c["nj"] - 1, 2, c["nk"] - 1]))
    return {"case": c, "q": q, "dx": dx, "inv_j": inv_j, "ints": ints, "rhsi": np.zeros_like(q)}


def _run_flux(s):
    base, g = ctypes.addressof(s["ints"]), ctypes.c_double(GAMMA)
    arrays = [ctypes.c_void_p(s[n].ctypes.data) for n in ("rhsi", "q", "dx", "inv_j")]
    _lib.check(_lib.load().aero_inviscid_flux_1(*arrays, *[ctypes.c_void_p(base + 4 * n) for n in range(18)],
                                                ctypes.byref(g)), "inviscid_flux_1")
    return s["rhsi"]


def exact(case, seed):
    """The Roe flux on WENO3 states of the transient call.  The whole runs have
    no closed value: they iterate the scheme many times."""
    if case["kind"] != "flux":
        return None
    q, dx, inv_j = _flux_arrays(case, np.random.default_rng(seed))
    rhs = np.zeros_like(q)
    for d in range(3):
        ax = 2 - d
        f = _faces(np.moveaxis(q, ax, 0), np.moveaxis(dx, ax, 0)[..., 3 * d:3 * d + 3], np.moveaxis(inv_j, ax, 0))
        rhs += np.moveaxis(np.concatenate([0 * f[:1], f[:-1] - f[1:], 0 * f[:1]]), 0, ax)
    out = np.zeros_like(q)
    inner = (slice(1, -1),) * 3
    out[inner] = rhs[inner]
    return out


def _faces(q, m, inv_j):
    """Fluxes at the faces n + 1/2 along axis 0."""
    def mix(a, b, c):  # the WENO3 state beside b, upwind from a
        s1, s2 = 1 / (3 * (1e-6 + (b - a) ** 2) ** 2), 2 / (3 * (1e-6 + (c - b) ** 2) ** 2)
        return (s1 * (1.5 * b - 0.5 * a) + s2 * (0.5 * b + 0.5 * c)) / (s1 + s2)

    left, right = q[:-1].copy(), q[1:].copy()
    left[1:] = mix(q[:-2], q[1:-1], q[2:])
    right[:-1] = mix(q[2:], q[1:-1], q[:-2])
    mj = m * inv_j[..., None]
    k = 0.5 * (mj[:-1] + mj[1:])
    size = np.sqrt((k ** 2).sum(-1))
    n = k / size[..., None]

    def side(s):
        rho, vel = s[..., 0], s[..., 1:4] / s[..., :1]
        p = (s[..., 4] - 0.5 * rho * (vel ** 2).sum(-1)) * (GAMMA - 1)
        h, un = GAMMA * p / ((GAMMA - 1) * rho) + 0.5 * (vel ** 2).sum(-1), (vel * k).sum(-1)
        f = np.concatenate([(rho * un)[..., None], (rho * un)[..., None] * vel + k * p[..., None],
                            (rho * h * un)[..., None]], -1)
        return rho, vel, p, h, un, f

    rl, vl, pl, hl, ul, fl = side(left)
    rr, vr, pr, hr, ur, fr = side(right)
    t, rho = np.sqrt(rr / rl), np.sqrt(rl * rr)
    vel, h = (vl + vr * t[..., None]) / (1 + t[..., None]), (hl + hr * t) / (1 + t)
    c2 = (GAMMA - 1) * (h - 0.5 * (vel ** 2).sum(-1))
    c, un = np.sqrt(c2), (vel * n).sum(-1)

    def fix(lam):
        lam = np.abs(lam)
        return np.where(lam < 0.06, (lam ** 2 + 0.06 ** 2) / 0.12, lam)

    dp, du, dv = pr - pl, (ur - ul) / size, vr - vl
    a1 = fix(un) * (rr - rl - dp / c2)
    a2, a3 = fix(un + c) * (dp + rho * c * du) / (2 * c2), fix(un - c) * (dp - rho * c * du) / (2 * c2)
    a4, a5 = a1 + a2 + a3, c * (a2 - a3)
    am = fix(un)[..., None] * rho[..., None] * (dv - du[..., None] * n)
    e = h * a4 + un * a5 + (vel * am).sum(-1) - c2 * a1 / (GAMMA - 1)
    diss = np.concatenate([a4[..., None], vel * a4[..., None] + a5[..., None] * n + am, e[..., None]], -1)
    return 0.5 * (fl + fr - size[..., None] * diss)


# ----------------------------------------------------------------------- work
def _nodes(c):
    k = c["kind"]
    if k in ("bump", "crank", "flux"):
        return c["ni"] * c["nj"] * c["nk"]
    if k in ("naca", "dropin"):
        return c["nblk"] * c["ni"] * c["nj"] * c["nk"]
    if k == "plate":
        nb = (c["nbi"], c["nbj"], c["nbk"])
        return math.prod((n - 1 + b) for n, b in zip((c["ni"], c["nj"], c["nk"]), nb))
    if k == "family":
        return c["members"] * 4 * c["ni"] * c["nj"] * c["nk"]
    rng = np.random.default_rng(c["sweep"])
    total = 0
    for _ in range(c["ncase"]):
        total += int(rng.integers(65, 258)) * int(rng.integers(33, 98)) * 5
        rng.uniform(0.05, 0.12), rng.uniform(0.3, 0.7)
    return total


def work(case):
    """Bytes: per node and iteration the solution, the metrics and 1/J read and
    the solution written (SA: nu_t and the wall distance as well), each field
    once.  Operations: of the network, its matrix products."""
    c = case
    if c["kind"] == "mlp":
        w, d = c["width"], c["depth"]
        per_row = 2.0 * (9 * w + (d - 1) * w * w + 5 * w)
        rows = 3 * c["batch"] * c["steps"] + c["predict"]
        params = 9 * w + (d - 1) * w * w + 5 * w
        return {"bytes": c["batch"] * c["steps"] * 14 * 4 + c["predict"] * 14 * 4 + 24 * params * c["steps"],
                "flops": per_row * rows}
    n = _nodes(c)
    if c["kind"] == "flux":
        return {"bytes": n * 8 * 20, "flops": n * 3 * 300}
    sa = c["kind"] in ("plate", "family") or bool(c.get("sa"))
    words = 20 + (3 if sa else 0) + (20 if c["kind"] == "crank" else 0)
    return {"bytes": n * 8.0 * words * c["iters"], "flops": 0}
