"""What a user of this library has it compute, as measurable cases.

Every case goes through the public binding (``ttifd.Modeling``, ``ttifd.Batch``):

``shot``      one shot on a handle whose model is uploaded: source and receiver
              geometry, the whole time loop, the traces fetched.
``program``   what one drop-in program run does: create, upload of the physical
              model, geometry, the time loop with snapshots, traces, destroy.
``batch``     many shots of one model, or many models of different sizes,
              advanced together.
``gradient``  one iteration of an inversion for one shot: the new model
              uploaded, the adjoint-state gradient, the four gradients and the
              source gradient fetched.
``batch_gradient``  the gradients of many shots of one model at once.

Sizes follow the repository's own configurations (layered 200 x 400 and
600 x 1200, the salt-like 1126 x 7872 and its 1126 x 3000 crop, models of
256-1126 x 256-4096 in one batch) with shorter time axes, plus ragged sizes.
``exact`` restates the scheme (rotated staggered grid, MEAL rims, image free
surface, the three rotations) in 64 bits with torch; gradients come from
automatic differentiation of that restatement.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("tti-fdmodeling_b200"))
import ttifd  # noqa: E402

VARIANTS = ("coordinate_rotation", "tensor_rotation", "bond_transformation")
DT = 0.0008


def listed():
    return [
        # a first look at a set-up: a few cells, launch latency only
        _case("shot", "shot_tiny_60x80", 0, 60, 80, 400, fpeak=25.0, eal=10, fs=1, seistype=3),
        # the small layered model of the parity configurations, whole time axis
        _case("shot", "shot_layered_200x400", 0, 200, 400, 1501, fpeak=15.0, eal=40, fs=0, seistype=1),
        # ragged mid-size grid, unequal spacing, a body-force source, every second sample recorded
        _case("shot", "shot_tensor_401x857", 1, 401, 857, 500, dz=8.0, fpeak=18.0, eal=30, fs=0, stype=6, seistype=3,
              mt=2),
        # the gradient workload's grid, forward only, free surface
        _case("shot", "shot_bond_600x1200", 2, 600, 1200, 400, fpeak=15.0, eal=40, fs=1, seistype=1),
        # the full demo grid, every column a receiver
        _case("shot", "shot_salt_1126x7872", 0, 1126, 7872, 150, fpeak=12.0, eal=60, fs=1, seistype=3),
        # one program run on the crop of the demo grid: set-up, snapshots and traces included
        _case("program", "program_tensor_1126x3000", 1, 1126, 3000, 150, fpeak=12.0, eal=50, fs=1, seistype=3, wsave=2,
              snap=75),
        # a survey's shots over one model
        _case("batch", "batch_16shots_1126x3000", 0, 1126, 3000, 40, fpeak=12.0, eal=50, fs=1, seistype=1, shots=16),
        # independent models of different sizes together
        _case("batch", "batch_models_uneven", 0, 1126, 4096, 60, fpeak=15.0, eal=40, fs=0, seistype=1, models=12),
        # inversion, every step kept
        _case("gradient", "gradient_600x1200_kept", 0, 600, 1200, 300, fpeak=15.0, eal=40, fs=1, seistype=1, ncheck=1),
        # inversion with checkpoints on a ragged grid, tensor rotation, pressure data
        _case("gradient", "gradient_tensor_233x517", 1, 233, 517, 300, fpeak=20.0, eal=25, fs=0, seistype=2, ncheck=10),
        # a large inversion shot that has to recompute, Bond transformation
        _case("gradient", "gradient_bond_1126x3000", 2, 1126, 3000, 60, fpeak=15.0, eal=50, fs=1, seistype=3, ncheck=6),
        # the shots of one inversion iteration together, binomial checkpoints
        _case("batch_gradient", "batch_gradient_8x300x600", 0, 300, 600, 200, fpeak=18.0, eal=30, fs=1, seistype=1,
              shots=8, ncheck=10),
    ]


def _case(kind, name, variant, nz, nx, nt, dz=10.0, fpeak=15.0, eal=30, fs=0, stype=1, seistype=1, mt=1, shots=1,
          models=1, ncheck=1, wsave=0, snap=1):
    c = dict(kind=kind, variant=VARIANTS[variant], nz=nz, nx=nx, nt=nt, dx=10.0, dz=dz, fpeak=fpeak, ealThick=eal,
             freesurface=fs, stype=stype, seistype=seistype, mt=mt, shots=shots, models=models, ncheck=ncheck,
             wsave=wsave, snap_sample=snap)
    return dict(c, name=name) if name else c


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("shot", "shot", "shot", "program", "batch", "batch", "gradient", "gradient", "batch_gradient"))
    o = dict(dz=rng.choice((10.0, 10.0, 8.0, 12.5)), fpeak=rng.uniform(12.0, 25.0), eal=rng.randint(10, 60),
             fs=rng.randint(0, 1), stype=rng.choice((1, 1, 1, 2, 4, 5, 6, 7, 8)), seistype=rng.choice((1, 1, 2, 3)),
             mt=rng.choice((1, 1, 1, 2, 4)))
    v = rng.choice((0, 0, 1, 2))
    if kind == "shot":
        nz, nx = _log(rng, 50, 1200), _log(rng, 60, 8000)
        work = 4.0e8
    elif kind == "program":
        nz, nx = _log(rng, 100, 1200), _log(rng, 100, 4000)
        o.update(wsave=rng.choice((1, 2, 3)))
        work = 3.0e8
    elif kind == "batch":
        o["stype"] = rng.choice((1, 1, 3, 6))
        if rng.random() < 0.5:
            o.update(shots=rng.randint(4, 24))
            nz, nx = _log(rng, 100, 1200), _log(rng, 100, 3000)
        else:
            o.update(models=rng.randint(4, 14))
            nz, nx = rng.randint(400, 1126), rng.randint(600, 4096)
        work = 5.0e8
    elif kind == "gradient":
        o.update(ncheck=rng.choice((1, 4, 8, 12)))
        nz, nx = _log(rng, 80, 1000), _log(rng, 100, 2500)
        work = 1.2e8
    else:
        o.update(shots=rng.randint(3, 10), ncheck=rng.choice((4, 8, 12)))
        nz, nx = _log(rng, 100, 500), _log(rng, 120, 900)
        work = 1.2e8
    cells = (nz + 2 * o["eal"] + 10) * (nx + 2 * o["eal"] + 10) * o.get("shots", 1) * (o.get("models", 1) * 0.5 + 0.5)
    nt = max(40, min(800, int(work / cells)))
    if kind == "program":
        o["snap"] = max(20, nt // 3)
    if kind in ("gradient", "batch_gradient") and o["ncheck"] == 1:
        nt = min(nt, 250)
    return _case(kind, None, v, nz, nx, nt, **o)


# ---------------------------------------------------------------- inputs
def _model(rng, nz, nx):
    """vp, vs, rho, epsilon, delta, theta of a dipping layered medium with an
    isotropic high-velocity body, physical (nx, nz) float32."""
    n = int(rng.integers(8, 25))
    x = torch.arange(nx, dtype=torch.float32)[:, None]
    z = torch.arange(nz, dtype=torch.float32)[None, :]
    a, wl, ph = rng.uniform(0.01, 0.04) * nz, rng.uniform(0.4, 1.2) * nx, rng.uniform(0, 2 * math.pi)
    slope = rng.uniform(-0.05, 0.05)
    relief = slope * (x - nx / 2) + a * torch.sin(2 * math.pi * x / wl + ph)
    dip = torch.rad2deg(torch.atan(slope + a * 2 * math.pi / wl * torch.cos(2 * math.pi * x / wl + ph)))
    li = ((z + relief) * (n / nz)).clamp(0, n - 1).to(torch.int64)
    body = ((x - nx * rng.uniform(0.35, 0.65)) / (0.12 * nx)) ** 2 + ((z - nz * 0.6) / (0.15 * nz)) ** 2 <= 1.0
    vt = np.clip(np.linspace(1600, 4600, n) + rng.normal(0, 60, n), 1500, 4750)
    et = rng.uniform(0.02, 0.25, n)
    dt = et * rng.uniform(0.1, 0.9, n)
    tt = rng.uniform(-15, 15, n)
    by = lambda t, inside: torch.tensor(t, dtype=torch.float32)[li].masked_fill_(body, inside)  # noqa: E731
    vp = by(vt, 4500.0)
    theta = (by(tt, 0.0) + dip).masked_fill_(body, 0.0)
    f = (vp, vp / 1.8, 310.0 * vp.sqrt().sqrt(), by(et, 0.0), by(dt, 0.0), theta)
    return [t.contiguous().numpy() for t in f]


def _ricker(nt, fpeak, amp):
    t = np.arange(nt) * DT - 1.0 / fpeak
    a = (np.pi * fpeak * t) ** 2
    return (amp * (1.0 - 2.0 * a) * np.exp(-a)).astype(np.float32)


def _observed(rng, n, nts, mt, fpeak, scale):
    """Recorded data of a line of n receivers: hyperbolic events and noise."""
    t = np.arange(nts, dtype=np.float32)[None, :] * np.float32(DT * mt)
    off = np.abs(np.arange(n, dtype=np.float32) - n * rng.uniform(0.3, 0.7))[:, None] * 10.0
    d = rng.standard_normal((n, nts)).astype(np.float32) * np.float32(0.02)
    for _ in range(4):
        t0, v = rng.uniform(0.03, 0.2), rng.uniform(1600, 4000)
        a = (np.float32(np.pi * fpeak) * (t - np.sqrt(t0 * t0 + (off / v) ** 2))) ** 2
        d += np.float32(rng.uniform(-1, 1)) * (1 - 2 * a) * np.exp(-np.minimum(a, 60.0))
    return (d * np.float32(scale)).astype(np.float32)


def _geometry(rng, case, nz, nx, shot=0):
    """(source columns, source rows, wavelets, receiver columns, receiver rows)"""
    sx = int(nx * (0.3 + 0.4 * (shot % case["shots"] + rng.random()) / case["shots"]))
    sz = 2 if case["freesurface"] else min(nz - 1, 8 + int(rng.integers(0, 8)))
    w = _ricker(case["nt"], case["fpeak"], rng.uniform(0.5, 2.0))[None, :]
    return [sx], [sz], w, np.arange(nx, dtype=np.int32), 2 + (0 if case["freesurface"] else 3)


def _kinds(seistype):
    return {1: (0, 1), 2: (2,), 3: (0, 1, 2)}[seistype]


def _config(case, nz=None, nx=None, nt=None):
    keys = ("variant", "dx", "dz", "fpeak", "ealThick", "freesurface", "stype", "seistype", "mt", "wsave",
            "snap_sample")
    return dict({k: case[k] for k in keys}, nz=nz or case["nz"], nx=nx or case["nx"], nt=nt or case["nt"], dt=DT)


def _rng(case, seed):
    return np.random.default_rng([seed, case["nz"], case["nx"], case["nt"]])


def _sizes(case):
    """Grids and time axes of a batch's models (the first is the case's own)."""
    r = np.random.default_rng([case["nz"], case["nx"], case["models"]])
    s = [(case["nz"], case["nx"], case["nt"])]
    for _ in range(case["models"] - 1):
        s.append((int(r.integers(256, max(257, case["nz"]) + 1)), int(r.integers(256, max(257, case["nx"]) + 1)),
                  int(r.integers(max(1, case["nt"] // 2), case["nt"] + 1))))
    return s


def _pad(fields, case):
    e = case["ealThick"] + 5
    return [np.pad(f, e, mode="edge") for f in fields]


def _data(rng, case, k, n):
    """Observed traces of component k at the amplitude of the source's own."""
    nts = (case["nt"] - 1) // case["mt"] + 1
    v, p = (5e-12, 4e-5) if case["stype"] == 1 else (3.0, 2e6) if case["stype"] == 8 else (1e-5, 40.0)
    return _observed(rng, n, nts, case["mt"], case["fpeak"], p if k == 2 else v)


def prepare(case, seed):
    rng = _rng(case, seed)
    kind, kinds = case["kind"], _kinds(case["seistype"])
    nts = (case["nt"] - 1) // case["mt"] + 1
    st = dict(case=case, kinds=kinds)
    if kind in ("shot", "gradient"):
        m = _model(rng, case["nz"], case["nx"])
        geo = _geometry(rng, case, case["nz"], case["nx"])
        h = ttifd.Modeling(device=0, **_config(case))
        st.update(h=h, geo=geo)
        if kind == "shot":
            h.upload_model_physical(*m)
            st["out"] = [ttifd.host_empty((case["nx"], nts)) for _ in kinds]
        else:
            st["model"] = m
            h.upload_model_physical(*m)
            _set(h, geo, kinds)
            for k in kinds:
                h.grad_set_observed(k, _data(rng, case, k, case["nx"]))
    elif kind == "program":
        m = _model(rng, case["nz"], case["nx"])
        st["model"] = [ttifd.host_empty(a.shape) for a in m]
        for d, a in zip(st["model"], m):
            d[...] = a
        st["geo"] = _geometry(rng, case, case["nz"], case["nx"])
        nk = {1: 2, 2: 1, 3: 3}[case["wsave"]]
        st["snap"] = ttifd.host_empty(nk * case["nz"] * case["nx"])
        nsnap = (case["nt"] - 1) // case["snap_sample"] + 1
        st["snaps"] = np.zeros((nsnap, nk, case["nx"], case["nz"]), np.float32)
        st["out"] = [ttifd.host_empty((case["nx"], nts)) for _ in kinds]
    else:
        sizes = _sizes(case)
        model_of = list(range(len(sizes))) if case["models"] > 1 else [0] * case["shots"]
        b = ttifd.Batch([_config(case, *s) for s in sizes], model_of, device=0)
        for i, (nz, nx, _) in enumerate(sizes):
            b.upload_model(i, *_pad(_model(rng, nz, nx), case))
        st.update(b=b, geo=[], out=[])
        for i, mo in enumerate(model_of):
            nz, nx, nt = sizes[mo]
            g = _geometry(rng, dict(case, nt=nt), nz, nx, i)
            st["geo"].append(g)
            if kind == "batch":
                n = (nt - 1) // case["mt"] + 1
                st["out"].append([ttifd.host_empty((nx, n)) for _ in kinds])
            else:
                _set(b.instances[i], g, kinds)
                for k in kinds:
                    b.instances[i].grad_set_observed(k, _data(rng, case, k, nx))
    return st


def _set(h, geo, kinds):
    sx, sz, w, gx, gz = geo
    h.set_source(sx, sz, w)
    for k in kinds:
        h.set_receivers(k, gx, gz)


def run(state):
    case, kinds = state["case"], state["kinds"]
    kind = case["kind"]
    if kind == "shot":
        h = state["h"]
        _set(h, state["geo"], kinds)
        h.run()
        return [h.fetch_traces(k, out=o) for k, o in zip(kinds, state["out"])]
    if kind == "program":
        with ttifd.Modeling(device=0, **_config(case)) as h:
            h.upload_model_physical(*state["model"])
            _set(h, state["geo"], kinds)
            h.set_snapshot_buffer(state["snap"])
            got = []

            def keep(it, which, a):
                state["snaps"][it // case["snap_sample"], len(got) % state["snaps"].shape[1]] = a
                got.append(which)

            h.run(keep, copy=False)
            return dict(traces=[h.fetch_traces(k, out=o) for k, o in zip(kinds, state["out"])], snaps=state["snaps"])
    if kind == "batch":
        b = state["b"]
        for inst, g in zip(b.instances, state["geo"]):
            _set(inst, g, kinds)
        b.run()
        return [inst.fetch_traces(k, out=o) for inst, out in zip(b.instances, state["out"]) for k, o in zip(kinds, out)]
    if kind == "gradient":
        h = state["h"]
        h.upload_model_physical(*state["model"])
        h.grad_zero()
        j = h.grad_run(case["ncheck"])
        return dict(J=j, source=h.grad_fetch_source(1), **{g: h.grad_fetch(g) for g in ("vp", "eps", "delta", "theta")})
    b = state["b"]
    b.instances[0].grad_zero()
    keep = -(-case["nt"] // case["ncheck"])
    j = b.grad_run(case["ncheck"] - 1, keep)
    return dict(J=np.array(j), source=np.stack([i.grad_fetch_source(1) for i in b.instances]),
                **{g: b.instances[0].grad_fetch(g) for g in ("vp", "eps", "delta", "theta")})


def work(case):
    """State read and written once and parameters read once per cell and step
    (a batch's shots share their model's parameters); a gradient adds one
    reverse step per forward step that reads and writes the adjoint state and
    the gradient sums and reads the parameters and the state of the forward
    step. The stencils alone: 2 x 28 operations per field and half-step."""
    f = 8 if case["variant"] == VARIANTS[1] else 5
    par = {VARIANTS[0]: 44, VARIANTS[1]: 40, VARIANTS[2]: 36}[case["variant"]]
    e = 2 * (case["ealThick"] + 5)
    nbytes = flops = 0.0
    for nz, nx, nt in (_sizes(case) if case["models"] > 1 else [(case["nz"], case["nx"], case["nt"])]):
        n = (nz + e) * (nx + e)
        nbytes += n * nt * (8.0 * f * case["shots"] + par)
        flops += n * nt * case["shots"] * 180.0
        if case["kind"] in ("gradient", "batch_gradient"):
            nbytes += n * nt * case["shots"] * (8.0 * f + 4.0 * 5 + 8.0 * 6 + par)
            flops += n * nt * case["shots"] * 260.0
        nbytes += 4.0 * nx * nt * len(_kinds(case["seistype"])) * case["shots"]
        if case["kind"] == "program":
            nbytes += 24.0 * nz * nx + 84.0 * n
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------- 64 bits
_C = (1.24362739770907, -0.114021164233934, 0.0272965993810630, -0.00699199493927320, 0.00132022981661381)


class _Exact:
    """The scheme in float64: set-up from the float32 model, then time steps.
    `leaf`: vp, epsilon, delta and theta carry gradients (vs, rho and the MEAL
    arrays held fixed)."""

    def __init__(self, case, model, leaf=False):
        self.case = case
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.e = case["ealThick"] + 5
        self.fs, self.v = case["freesurface"], VARIANTS.index(case["variant"])
        pads = [np.pad(f, self.e, mode="edge") for f in model]
        vp, vs, rho, eps, delta, theta = (torch.tensor(p, dtype=torch.float64, device=self.dev) for p in pads)
        self.leaves = None
        if leaf:
            self.leaves = [t.requires_grad_() for t in (vp, eps, delta, theta)]
        self.nx, self.nz = vp.shape
        self.i0 = self.e if self.fs else 5
        dx, dz = case["dx"], case["dz"]
        f32 = lambda x: float(np.float32(x))  # noqa: E731
        self.ihx, self.ihz, self.dt = 0.5 * f32(1.0 / dx), 0.5 * f32(1.0 / dz), f32(DT)
        # MEAL: damping and velocity scaling rims
        vp0, n = vp.detach(), self.e
        iz = torch.arange(self.nz, device=self.dev)[None, :].expand(self.nx, -1)
        ix = torch.arange(self.nx, device=self.dev)[:, None].expand(-1, self.nz)
        lz = torch.zeros_like(iz)
        if not self.fs:
            lz = torch.where(iz < n, n - iz, lz)
        lz = torch.where(iz >= self.nz - n, iz - (self.nz - n - 1), lz)
        row = iz >= (n if self.fs else 0)
        lx = torch.where(row & (ix < n), n - ix, torch.zeros_like(ix))
        lx = torch.where(row & (ix >= self.nx - n), ix - (self.nx - n - 1), lx)
        lr = math.log(10.0) * (-(math.log10(n) - 1.0) / math.log10(2.0) - 3.0 - 0.5 * 2)
        vss = torch.where(vs == 0, vp0 / math.sqrt(3.0), vs)
        d2, b2 = 0.0, 0.0
        for lay, h in ((lx, dx), (lz, dz)):
            w = torch.where(lay > 0, torch.exp(math.log(2.0) * (lay / n) ** 2.5) - 1.0, 0.0 * vp0)
            d2 = d2 + (-3.0 * vp0 * lr / (2.0 * n * h) * w) ** 2
            b2 = b2 + ((2.0 * vss / (h * f32(case["fpeak"])) / 10.0 - 1.0) * w) ** 2
        beta = torch.sqrt(b2) + 1.0
        hd = 0.5 * self.dt * torch.sqrt(d2) / beta
        c1, c2 = (1 - hd) / (1 + hd), self.dt / (1 + hd)
        p, s, r = vp / beta, vs / beta, rho * beta
        f = 1.0 - (s / p) ** 2
        c11 = r * p * p * (1 + 2 * eps)
        c13 = r * (p * p * torch.sqrt(f * (f + 2 * delta)) - s * s)
        c33, c55 = r * p * p, r * s * s
        th = theta * (math.pi / 180.0)
        sn, cs = torch.sin(th), torch.cos(th)
        s2t, c2t = torch.sin(2 * th), torch.cos(2 * th)

        def avg(a):
            return torch.nn.functional.pad(0.25 * (a[:-1, :-1] + a[1:, :-1] + a[:-1, 1:] + a[1:, 1:]), (0, 1, 0, 1))

        box = (slice(5, self.nx - 5), slice(self.i0, self.nz - 5))
        b = lambda a: a[box]  # noqa: E731
        self.box, self.c1, self.br, self.c2 = box, b(c1), b(c2 / avg(r).clamp_min(1e-30)), b(c2)
        self.snv, self.csv = b(avg(sn)), b(avg(cs))
        if self.v == 2:
            x2, y2, u = sn * sn, cs * cs, c13 + 2 * c55
            b11 = c11 * y2 * y2 + c33 * x2 * x2 + (0.5 * c13 + c55) * s2t ** 2
            b13 = (0.25 * (c11 + c33) - c55) * s2t ** 2 + c13 * (x2 * x2 + y2 * y2)
            b15 = 0.5 * (-c11 * y2 + c33 * x2 + u * c2t) * s2t
            b33 = c11 * x2 * x2 + c33 * y2 * y2 + (0.5 * c13 + c55) * s2t ** 2
            b35 = 0.5 * (-c11 * x2 + c33 * y2 - u * c2t) * s2t
            b55 = 0.25 * (c11 + c33 - 2 * c13) * s2t ** 2 + c55 * c2t ** 2
            m = [b11, b13, b15, b33, b35, b55]
            if self.fs:
                a11, a13, a15, a33, a35, a55 = (t[:, self.e:self.e + 1] for t in m)
                n35 = -(a13 * a55 - a15 * a35) / (a33 * a55 - a35 * a35)
                n55 = (a13 * n35 - a15 * a33) / (a33 * a55 - n35 * n35)
                rows = [a11 - a13 * n35 + a15 * n55] + [torch.zeros_like(a11)] * 5
                m = [torch.cat([t[:, :self.e], q, t[:, self.e + 1:]], 1) for t, q in zip(m, rows)]
            self.m = [b(t) for t in m]
        else:
            self.m = [b(t) for t in (c11, c13, c33, c55)]
        self.sn, self.cs, self.s2t = b(sn), b(cs), b(s2t)
        # the two diagonals of the stencil as 10 x 10 correlation kernels
        w = torch.zeros(2, 1, 10, 10, dtype=torch.float64)
        for k in range(1, 6):
            w[0, 0, k + 4, k + 4] += _C[k - 1]
            w[0, 0, 5 - k, 5 - k] -= _C[k - 1]
            w[1, 0, k + 4, 5 - k] += _C[k - 1]
            w[1, 0, 5 - k, k + 4] -= _C[k - 1]
        self.w = w.to(self.dev)
        h2 = dx * dx + dz * dz
        off = np.arange(-5, 6)
        rx, rz = off[:, None] * dx, off[None, :] * dz
        al = math.log(0.8) / h2
        g = np.exp(al * (rx * rx + rz * rz)) * f32(1 / dx) * f32(1 / dz) * self.dt
        t = lambda a: torch.tensor(a + 0.0 * g, dtype=torch.float64, device=self.dev)  # noqa: E731
        self.k = dict(g=t(g), kx=t(2 * al * rx * g), kz=t(2 * al * rz * g))

    def _diff(self, fields, at):
        """(d1, d2) of each field over the updated cells; at: 1 velocity nodes, 0 stress nodes"""
        o = torch.nn.functional.conv2d(torch.stack(fields)[:, None], self.w)
        x0, z0 = 5 - (4 if at else 5), self.i0 - (4 if at else 5)
        nx, nz = self.nx - 10, self.nz - 5 - self.i0
        return o[:, :, x0:x0 + nx, z0:z0 + nz]

    def _put(self, a, new):
        a = a.clone()
        a[self.box] = new
        return a

    def _add(self, a, x, z, k):
        """a plus the 11 x 11 window k centred on (x, z), clipped to the grid"""
        xa, xb, za, zb = max(0, x - 5), min(self.nx, x + 6), max(0, z - 5), min(self.nz, z + 6)
        a = a.clone()
        a[xa:xb, za:zb] += k[xa - x + 5:xb - x + 5, za - z + 5:zb - z + 5]
        return a

    def _vsource(self, vx, vz, x, z, s):
        st, k = self.case["stype"], self.k
        if st in (2, 4):
            vx, vz = self._add(vx, x, z, k["kx"] * s), self._add(vz, x, z, k["kz"] * s)
        if st in (3, 4):
            vx, vz = self._add(vx, x, z, -k["kz"] * s), self._add(vz, x, z, k["kx"] * s)
        if st == 5:
            vx = self._add(vx, x, z, k["g"] * s)
        if st == 6:
            vz = self._add(vz, x, z, k["g"] * s)
        if st == 7:
            q = 0.5 * math.sqrt(2.0) * s
            vx, vz = self._add(vx, x, z, k["g"] * q), self._add(vz, x, z, k["g"] * q)
        if st == 8:
            q = 0.125 * math.sqrt(2.0) * s
            vx, vz = vx.clone(), vz.clone()
            for ox, oz, gx, gz in ((0, 0, -1, 1), (-1, 0, -1, -1), (-1, -1, 1, -1), (0, -1, 1, 1)):
                vx[x + ox, z + oz] += gx * q
                vz[x + ox, z + oz] += gz * q
        return vx, vz

    def run(self, geo, snaps=None):
        c = self.case
        sx, sz, wav, gx, gz = geo
        x, z = sx[0] + self.e, sz[0] + self.e
        wav = torch.tensor(wav[0], dtype=torch.float64, device=self.dev)
        if self.leaves is not None:
            wav.requires_grad_()
            self.wav = wav
        zero = torch.zeros(self.nx, self.nz, dtype=torch.float64, device=self.dev)
        vx = vz = xx = zz = xz = tx = tz = tq = zero
        rx, rz = torch.tensor(np.asarray(gx) + self.e, device=self.dev), gz + self.e
        rec = {k: [] for k in _kinds(c["seistype"])}
        hx, hz, box = self.ihx, self.ihz, self.box
        for it in range(c["nt"]):
            d = self._diff([xx, zz, xz], 1)
            p, m = d[:, 0] + d[:, 1], d[:, 0] - d[:, 1]
            if self.v == 0:
                sv, cv = self.snv, self.csv
                fx = cv * hx * p[0] - sv * hx * m[0] + sv * hx * p[2] + cv * hz * m[2]
                fz = cv * hx * p[2] - sv * hz * m[2] + sv * hx * p[1] + cv * hz * m[1]
            else:
                fx, fz = hx * p[0] + hz * m[2], hx * p[2] + hz * m[1]
            vx = self._put(vx, self.c1 * vx[box] + self.br * fx)
            vz = self._put(vz, self.c1 * vz[box] + self.br * fz)
            if c["stype"] > 1:
                vx, vz = self._vsource(vx, vz, x, z, wav[it])
            d = self._diff([vx, vz], 0)
            a, q = hx * (d[0, 0] + d[0, 1]), hz * (d[0, 0] - d[0, 1])
            r, s = hx * (d[1, 0] + d[1, 1]), hz * (d[1, 0] - d[1, 1])
            if self.v == 2:
                b11, b13, b15, b33, b35, b55 = self.m
                sh = r + q
                n = [b11 * a + b13 * s + b15 * sh, b13 * a + b33 * s + b35 * sh, b15 * a + b35 * s + b55 * sh]
                xx, zz, xz = (self._put(o, self.c1 * o[box] + self.c2 * u) for o, u in zip((xx, zz, xz), n))
            elif self.v == 0:
                c11, c13, c33, c55 = self.m
                sn, cs = self.sn, self.cs
                a, q, r, s = cs * a - sn * q, sn * a + cs * q, cs * r - sn * s, sn * r + cs * s
                n = [c11 * a + c13 * s, c13 * a + c33 * s, c55 * (r + q)]
                xx, zz, xz = (self._put(o, self.c1 * o[box] + self.c2 * u) for o, u in zip((xx, zz, xz), n))
            else:
                c11, c13, c33, c55 = self.m
                s2, c2, st = self.sn ** 2, self.cs ** 2, self.s2t
                sh = q + r
                ex, ez = c2 * a + s2 * s - 0.5 * st * sh, s2 * a + c2 * s + 0.5 * st * sh
                eq = st * (a - s) + (c2 - s2) * sh
                n = [c11 * ex + c13 * ez, c13 * ex + c33 * ez, c55 * eq]
                u, w, y = (self.c1 * o[box] + self.c2 * t for o, t in zip((tx, tz, tq), n))
                tx, tz, tq = self._put(tx, u), self._put(tz, w), self._put(tq, y)
                xx = self._put(xx, c2 * u + s2 * w + st * y)
                zz = self._put(zz, s2 * u + c2 * w - st * y)
                xz = self._put(xz, -0.5 * st * (u - w) + (c2 - s2) * y)
            if self.fs:
                i, cols = self.i0, slice(5, self.nx - 5)
                xx, zz, xz = xx.clone(), zz.clone(), xz.clone()
                zz[cols, i] = 0.0
                xz[cols, i] = 0.0
                up, dn = slice(i - 5, i), slice(i + 1, i + 6)
                xx[cols, up] = 2.0 * xx[cols, i:i + 1] - xx[cols, dn].flip(1)
                zz[cols, up] = -zz[cols, dn].flip(1)
                xz[cols, up] = -xz[cols, dn].flip(1)
            if c["stype"] == 1:
                g = 0.5 * self.k["g"] * wav[it]
                xx, zz = self._add(xx, x, z, g), self._add(zz, x, z, g)
                if self.v == 1:
                    tx, tz = self._add(tx, x, z, g), self._add(tz, x, z, g)
            if it % c["mt"] == 0:
                for k in rec:
                    rec[k].append(vx[rx, rz] if k == 0 else vz[rx, rz] if k == 1 else
                                  0.5 * (xx[rx, rz] + zz[rx, rz]))
            if snaps is not None and it % c["snap_sample"] == 0:
                e = self.e
                inner = (slice(e, self.nx - e), slice(e, self.nz - e))
                f = {1: vx, 2: vz, 3: 0.5 * (xx + zz)}
                snaps.append(torch.stack([f[k][inner] for k in {1: (1, 2), 2: (3,), 3: (1, 2, 3)}[c["wsave"]]]))
        return [torch.stack(v, 1) for v in rec.values()]


def exact(case, seed):
    e = 2 * (case["ealThick"] + 5)
    cells = float((case["nz"] + e) * (case["nx"] + e)) * case["shots"]
    rng = _rng(case, seed)
    kinds = _kinds(case["seistype"])
    host = lambda t: t.detach().cpu().numpy()  # noqa: E731
    if case["kind"] in ("gradient", "batch_gradient"):
        # automatic differentiation keeps every step
        if cells * case["nt"] > 1.0e8 or cells / case["shots"] * case["nt"] > 6.0e7:
            return None
        m = _model(rng, case["nz"], case["nx"])
        jobs = []
        for i in range(case["shots"]):
            g = _geometry(rng, case, case["nz"], case["nx"], i)
            jobs.append((g, [_data(rng, case, k, case["nx"]) for k in kinds]))
        js, src, tot = [], [], None
        for g, obs in jobs:
            x = _Exact(case, m, leaf=True)
            tr = x.run(g)
            obs = [torch.tensor(o, dtype=torch.float64, device=x.dev) for o in obs]
            j = sum(0.5 * ((t - o) ** 2).sum() for t, o in zip(tr, obs))
            gr = torch.autograd.grad(j, x.leaves + [x.wav])
            js.append(float(j.detach()))
            src.append(host(gr[4])[None, :])
            tot = list(gr[:4]) if tot is None else [a + b for a, b in zip(tot, gr)]
        out = dict(zip(("vp", "eps", "delta", "theta"), (host(t) for t in tot)))
        if case["kind"] == "gradient":
            return dict(J=js[0], source=src[0], **out)
        return dict(J=np.array(js), source=np.stack(src), **out)
    if cells * case["models"] * case["nt"] > 4.0e8:
        return None
    with torch.no_grad():
        if case["kind"] == "batch":
            sizes = _sizes(case)
            ms = [_model(rng, nz, nx) for nz, nx, _ in sizes]
            out = []
            for i in range(max(case["models"], case["shots"])):
                mo = i if case["models"] > 1 else 0
                nz, nx, nt = sizes[mo]
                c = dict(case, nz=nz, nx=nx, nt=nt)
                out += [host(t) for t in _Exact(c, ms[mo]).run(_geometry(rng, c, nz, nx, i))]
            return out
        m = _model(rng, case["nz"], case["nx"])
        snaps = [] if case["kind"] == "program" else None
        tr = [host(t) for t in _Exact(case, m).run(_geometry(rng, case, case["nz"], case["nx"]), snaps)]
        return tr if snaps is None else dict(traces=tr, snaps=host(torch.stack(snaps)))
