"""The work that a user of the library has it do, as cases to measure: time loops of single
channels in both precisions, of a bounded flow over a step, of an ensemble and of a channel with
the learned closure; the closure's training and its training data; the statistics of a running
channel.

A case is a dict of plain values.  prepare() makes what a program has in hand before the call
(contexts with an uploaded state, datasets, networks), run() is one pass through the public
calls, work() the bytes and operations a pass cannot do without, and exact() what run() returns
for a freshly prepared state, in 64 bits with plain torch.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "ark-cpp-mpi_gb300"))

import arkgpu  # noqa: E402

F64 = torch.float64
CHANNEL = (2 * math.pi, 2.0, math.pi)  # the channel's box
SOUND, RHO0, CFL = 10.0, 1.0, 0.2
ENSEMBLE_GRIDS = ((32, 32, 32), (64, 32, 32), (64, 48, 48), (96, 64, 64), (128, 64, 64))
U_TAU = 0.05  # friction velocity the closure's y+ is taken with
CELLS = ("ronCon", "u1nCon", "u2nCon", "u3nCon")
FACES = tuple(f"{v}{d}" for d in "123" for v in ("p", "u1", "u2", "u3"))


def listed():
    return [
        # a small FP64 run that must agree with the reference bit for bit (100 of its steps at a time)
        dict(name="fp64 64x32x32", kind="flow", c1=64, c2=32, c3=32, fp64=True, steps=100, re=2800.0),
        # the benchmark channel in FP64 as one job: state up, steps, state down
        dict(name="fp64 job 256x128x128", kind="flow", c1=256, c2=128, c3=128, fp64=True, steps=40, re=5600.0, job=True),
        # the reference's own program: flow over a backward-facing step, bounded in x and z, one layer of cells
        dict(name="fp64 step 200x60x1", kind="flow", c1=200, c2=60, c3=1, fp64=True, steps=200, re=1000.0, step=True),
        # the throughput path at its largest grid, between two looks at the state
        dict(name="fp32 512x256x256", kind="flow", c1=512, c2=256, c3=256, fp64=False, steps=100, re=5600.0),
        # the fine run of the closure study
        dict(name="fp32 256x128x128", kind="flow", c1=256, c2=128, c3=128, fp64=False, steps=100, re=5600.0),
        # its coarse run
        dict(name="fp32 64x48x48", kind="flow", c1=64, c2=48, c3=48, fp64=False, steps=200, re=5600.0),
        # an odd-sized FP32 grid, bounded in x and z, as a job of a few steps
        dict(name="fp32 job 150x67x93 bounded", kind="flow", c1=150, c2=67, c3=93, fp64=False, steps=50, re=3000.0,
             bounded=True, job=True),
        # 64 channels of mixed sizes and Reynolds numbers side by side
        dict(name="ensemble 64", kind="ensemble", members=64, steps=100),
        # the coarse run with the learned closure on
        dict(name="closure 64x48x48", kind="flow", c1=64, c2=48, c3=48, fp64=False, steps=200, re=5600.0, closure=True),
        # an epoch of the closure's training
        dict(name="train 2097152 rows", kind="train", rows=1 << 21, batch=65536),
        # training data of one snapshot of the fine run
        dict(name="samples 256x128x128", kind="samples", c1=256, c2=128, c3=128, stride=4, fp64=False),
        # the statistics of a running channel: profile, plane moments, conservation sums, energy
        dict(name="statistics 256x128x128", kind="statistics", c1=256, c2=128, c3=128, fp64=False),
    ]


def _size(rng, lo, hi):
    """A size between lo and hi, spread over its logarithm; a third of them whole multiples of 16."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, n // 16 * 16) if rng.random() < 1 / 3 else n


def draw(rng):
    kind = rng.choice(["fp64", "fp64", "step", "fp32", "fp32", "fp32", "ensemble", "closure", "train", "samples",
                       "statistics"])
    grid = lambda big: dict(c1=_size(rng, 16, 512 if big else 256), c2=_size(rng, 16, 256 if big else 128),
                            c3=_size(rng, 16, 256 if big else 128))
    cells = lambda c: c["c1"] * c["c2"] * c["c3"]
    steps = lambda c, most: int(max(20, min(200, most / cells(c))))
    if kind in ("fp64", "fp32"):
        c = dict(kind="flow", **grid(kind == "fp32"))
        c.update(fp64=kind == "fp64", steps=steps(c, 1.6e8 if kind == "fp64" else 2.5e9), re=round(rng.uniform(2000, 6000)))
        if rng.random() < 0.25:
            c.update(bounded=True, job=True, steps=20)
        return c
    if kind == "step":
        return dict(kind="flow", c1=_size(rng, 60, 400), c2=_size(rng, 30, 120), c3=rng.choice([1, 1, 2, 5]), fp64=True,
                    steps=100, re=1000.0, step=True)
    if kind == "ensemble":
        return dict(kind="ensemble", members=_size(rng, 4, 64), steps=rng.choice([30, 60, 100]))
    if kind == "closure":
        c = dict(kind="flow", **{a: _size(rng, 24, b) for a, b in (("c1", 128), ("c2", 64), ("c3", 64))})
        return dict(c, fp64=False, steps=100, re=5600.0, closure=True)
    if kind == "train":
        batch = 1 << rng.randint(12, 16)
        return dict(kind="train", rows=batch * rng.randint(8, 32) + rng.randint(0, batch - 1), batch=batch)
    c = dict(kind=kind, **grid(False), fp64=rng.random() < 0.3)
    return dict(c, stride=rng.choice([1, 2, 4, 8])) if kind == "samples" else c


# ---- inputs ----------------------------------------------------------------------------------

def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _box(case):
    """The lengths of the domain: the channel's, or those of the backward-facing step (layers of 0.1)."""
    return (20.0, 6.0, 0.1 * case["c3"]) if case.get("step") else CHANNEL


def _fluid(c1, c2, c3, step):
    """Interior cells that are fluid: all, or all but the block of a backward-facing step."""
    a = torch.ones(c3, c2, c1, dtype=torch.bool, device=_dev())
    if step:
        a[:, : max(1, c2 // 6), : max(1, c1 // 4)] = False
    return a


def _heights(c2):
    """The y of the channel's cell rows."""
    return -0.5 * CHANNEL[1] + (torch.arange(c2, dtype=F64, device=_dev()) + 0.5) * (CHANNEL[1] / c2)


def _velocity(seed, c1, c2, c3, amp, step):
    """Interior velocities [3, k, j, i]: a laminar channel profile (or the uniform inflow of the step) plus seeded
    uniform noise, at rest in solids."""
    g = torch.Generator(device=_dev()).manual_seed(seed)
    u = amp * (2 * torch.rand(3, c3, c2, c1, dtype=F64, device=_dev(), generator=g) - 1)
    y = _heights(c2)
    u[0] += 1.0 if step else 1.5 * (1 - y * y)[None, :, None]
    return u * _fluid(c1, c2, c3, step)


def _ghosted(a, px, pz):
    """Interior [..., k, j, i] with one layer around it: periodic images or copies in x and z, zeros beyond the walls."""
    a = torch.cat((a[..., -1:], a, a[..., :1]) if px else (a[..., :1], a, a[..., -1:]), -1)
    a = torch.cat((a[..., -1:, :, :], a, a[..., :1, :, :]) if pz else (a[..., :1, :, :], a, a[..., -1:, :, :]), -3)
    z = torch.zeros_like(a[..., :1, :])
    return torch.cat((z, a, z), -2)


def _faces(u, fluid, px, pz):
    """Velocities on the faces normal to x, y, z: the mean of the two cells, at rest at walls and solids."""
    g = _ghosted(u, px, pz)
    f = _solid(fluid, px, pz).logical_not()
    i = slice(1, -1)
    out = []
    for lo, hi in (((i, i, slice(0, -1)), (i, i, slice(1, None))), ((i, slice(0, -1), i), (i, slice(1, None), i)),
                   ((slice(0, -1), i, i), (slice(1, None), i, i))):
        a, b = (Ellipsis,) + lo, (Ellipsis,) + hi
        out.append(0.5 * (g[a] + g[b]) * (f[lo] & f[hi]))
    return out


def _solid(fluid, px, pz):
    """The solid cells with the ghost layer: the walls' rows, and a step's block continued into x and z ghosts."""
    s = _ghosted(fluid.to(F64), px, pz) < 0.5
    s[:, 0] = s[:, -1] = True
    return s


def _flow_params(c, re):
    lx, ly, lz = _box(c)
    p = arkgpu.make_params(c["c1"], c["c2"], c["c3"], re_b=re, sound=SOUND, rho0=RHO0, cfl=CFL, lx=lx, ly=ly, lz=lz,
                           precision=arkgpu.FP64 if c.get("fp64") else arkgpu.FP32,
                           forcing=not (c.get("step") or c.get("bounded")))
    if c.get("step") or c.get("bounded"):
        p.periodic_x = p.periodic_z = 0
    return p


_host = {}  # one page-locked host state per grid, as a program keeps one


def _host_state(p):
    key = (p.n1_cells, p.n2_cells, p.n3_cells)
    if key not in _host:
        _host[key] = arkgpu.PinnedState(p)
    return _host[key]


def _fill(h, p, u, fluid):
    """The host state of interior velocities u at rest density: both levels alike, faces between."""
    px, pz = p.periodic_x, p.periodic_z
    put = lambda name, a: torch.from_numpy(h.arrays[name]).copy_(a)
    g = _ghosted(u, px, pz)
    for lvl in ("", "n"):
        h.arrays[f"ro{lvl}Con"].fill(RHO0)
        for m in range(3):
            put(f"u{m + 1}{lvl}Con", g[m])
    put("condition", _solid(fluid, px, pz).to(F64))
    for d, f in enumerate(_faces(u, fluid, px, pz)):
        h.arrays[f"p{d + 1}"].fill(0.0)
        h.arrays[f"ro{d + 1}"].fill(RHO0)
        for m in range(3):
            full = torch.zeros(h.arrays["p1"].shape, dtype=F64, device=f.device)
            full[1:1 + f.shape[1], 1:1 + f.shape[2], 1:1 + f.shape[3]] = f[m]
            put(f"u{m + 1}{d + 1}", full)
    if torch.cuda.is_available():
        torch.cuda.synchronize()


def _inside(name, a):
    """The cells or faces of an array that a step defines (its last three axes)."""
    if name in CELLS:
        return a[..., 1:-1, 1:-1, 1:-1]
    e = [slice(1, -2)] * 3
    e[3 - int(name[-1])] = slice(1, -1)
    return a[(Ellipsis,) + tuple(e)]


def _ensemble_members(case, seed):
    """(grid, Reynolds number, noise, seed) of each member: the sizes are the case's, the rest the seed's."""
    sizes, r = np.random.default_rng(4242 + case["members"]), np.random.default_rng(seed)
    return [(ENSEMBLE_GRIDS[int(sizes.integers(len(ENSEMBLE_GRIDS)))], float(r.uniform(2000, 6000)),
             float(r.uniform(0.05, 0.15)), int(r.integers(1 << 40))) for _ in range(case["members"])]


def _network(seed):
    """Weights (every layer scaled by its inputs), and the mean and spread of the features."""
    r = np.random.default_rng(seed)
    w = np.concatenate([r.uniform(-1, 1, n) * s for n, s in
                        ((320, 0.55), (32, 0.0), (1024, 0.3), (32, 0.0), (32, 0.3), (1, 0.0))]).astype(np.float32)
    mu = np.array([0, 3, 2, 0, 0, 0, 0, 1, 1, 100], np.float32)
    sd = np.array([1, 2, 2, 1, 1, 1, 1, 1, 1, 80], np.float32)
    return w.astype(np.float64), mu.astype(np.float64), sd.astype(np.float64)


def _rows(case, seed):
    """Training rows as fine runs give them: signed invariants of mixed size, mostly small positive targets."""
    g = torch.Generator(device=_dev()).manual_seed(seed)
    x = torch.randn(case["rows"], 10, generator=g, device=_dev())
    scale = torch.tensor([0.1, 3, 2, 1, 1, 1, 0.7, 1, 1, 80.0], device=_dev())
    x = x * scale
    x[:, 1:3] = x[:, 1:3].abs()
    x[:, 9] = x[:, 9].abs()
    t = 0.05 * (x[:, 1] + x[:, 7] * x[:, 8]).clamp(min=0) + 0.02 * torch.rand(case["rows"], generator=g, device=_dev())
    return x, t


# ---- the calls -------------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        x, t = _rows(case, seed)
        data = arkgpu.ClosureData(case["rows"])
        data.append(x.cpu().numpy(), t.cpu().numpy())
        net = arkgpu.Mlp(seed=seed)
        net.set(*_network(seed))
        net.fit_normalization(data)
        return dict(case=case, data=data, net=net)
    if kind == "ensemble":
        members = _ensemble_members(case, seed)
        params = [_flow_params(dict(c1=c[0], c2=c[1], c3=c[2]), re) for c, re, _, _ in members]
        e = arkgpu.Ensemble(params)
        counts = {}
        for q, (c, _, amp, s) in enumerate(members):
            h = _host_state(params[q])
            _fill(h, params[q], _velocity(s, *c, amp, False), _fluid(*c, False))
            e.upload(q, h.arrays)
            counts[c] = counts.get(c, 0) + 1
        # where the fields of the members of one size come back to: side by side, page-locked
        out = {c: {f: torch.zeros(n, c[2] + 2, c[1] + 2, c[0] + 2, dtype=F64, pin_memory=torch.cuda.is_available()).numpy()
                   for f in CELLS} for c, n in sorted(counts.items())}
        at = {c: 0 for c in counts}
        host = []
        for c, *_ in members:
            host.append(arkgpu.host_struct({f: out[c][f][at[c]] for f in CELLS}))
            at[c] += 1
        return dict(case=case, ensemble=e, host=host, out=out)
    p = _flow_params(case, case.get("re", 5600.0))
    h = _host_state(p)
    size = (case["c1"], case["c2"], case["c3"])
    step = case.get("step", False)
    _fill(h, p, _velocity(seed, *size, 0.01 if step else 0.1, step), _fluid(*size, step))
    ctx = arkgpu.Context(p)
    s = dict(case=case, ctx=ctx, host=h)
    if case.get("job"):  # the host state goes up in every pass: this state's own copy of it
        s["start"] = arkgpu.PinnedState(p)
        s["start"].fill(h.arrays)
    ctx.upload_struct(h.struct())
    if case.get("closure"):
        s["net"] = arkgpu.Mlp(seed=seed)
        s["net"].set(*_network(seed))
        ctx.set_closure(s["net"], U_TAU)
    if kind == "samples":
        n = -(-size[0] // case["stride"]) * size[1] * -(-size[2] // case["stride"])
        s["data"] = arkgpu.ClosureData(n)
    return s


def _scalars(s):
    return {"dt": s.dt, "time": s.time, "nstep": int(s.nstep), "ub": s.bulk_velocity, "g": s.bulk_force}


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "flow":
        ctx = state["ctx"]
        if "start" in state:
            ctx.upload_struct(state["start"].struct())
        ctx.step(case["steps"])
        back = arkgpu.HostState()
        for n in CELLS + FACES:
            setattr(back, n, getattr(state["host"].h, n))
        ctx.download_struct(back)
        return {"scalars": _scalars(ctx.scalars()),
                "fields": {n: _inside(n, state["host"].arrays[n]) for n in CELLS + FACES}}
    if kind == "ensemble":
        e = state["ensemble"]
        e.step(case["steps"])
        for q, h in enumerate(state["host"]):
            if arkgpu.lib().ark_ensemble_download(e.h, q, ctypes.byref(h)) != 0:
                raise RuntimeError("ark_ensemble_download")
        return {f"{c[0]}x{c[1]}x{c[2]}": {n: _inside(n, a) for n, a in o.items()} for c, o in state["out"].items()}
    if kind == "train":
        loss = state["net"].train(state["data"], epochs=1, batch=case["batch"], lr=1e-3)
        return {"loss": loss, "weights": state["net"].get()[0].astype(np.float32)}
    if kind == "samples":
        state["data"].clear()
        state["ctx"].closure_sample(state["data"], sx=case["stride"], sz=case["stride"], u_tau=U_TAU)
        x, t = state["data"].get()
        return {"features": x, "targets": t}
    ctx = state["ctx"]
    prof, shear = ctx.mean_profile()
    s = ctx.sums()
    return {"profile": prof, "shear": shear, "planes": ctx.plane_stats(), "energy": ctx.kinetic_energy(),
            "sums": [s.mass, s.momentum1, s.momentum2, s.momentum3, s.kinetic], "cells": int(s.cells)}


def work(case):
    """The persistent state of a channel is 16 values a cell (density and velocity, and pressure and velocity on three
    faces), read and written by every step; what comes back to the host is written once more."""
    kind = case["kind"]
    if kind == "train":
        return {"bytes": case["rows"] * 44, "flops": case["rows"] * 6 * 1376}
    if kind == "ensemble":
        cells = sum(a * b * c for (a, b, c), *_ in _ensemble_members(case, 0))
        return {"bytes": case["steps"] * cells * 128 + cells * 32, "flops": case["steps"] * cells * 527}
    cells, word = case["c1"] * case["c2"] * case["c3"], 8 if case["fp64"] else 4
    if kind == "flow":
        moved = 16 * 8 + (24 * 8 if case.get("job") else 0)
        return {"bytes": cells * (case["steps"] * 32 * word + moved),
                "flops": cells * case["steps"] * (600 if case["fp64"] else 527 + 3000 * bool(case.get("closure")))}
    if kind == "samples":
        rows = -(-case["c1"] // case["stride"]) * case["c2"] * -(-case["c3"] // case["stride"])
        return {"bytes": cells * 3 * word + rows * 44, "flops": cells * 27 + rows * (6 * 27 + 400)}
    return {"bytes": cells * 4 * word, "flops": cells * 40}


# ---- the same in 64 bits ----------------------------------------------------------------------
# Interior arrays [member, k, j, i]; faces normal to x, y, z hold one more along their axis.  A
# step is as the scheme states it: time step, conservative half step with stress and forces, the
# characteristic face update of the three directions, the second half step.

DIM = (-1, -2, -3)  # the tensor axis of x, y, z


def _cut(a, d, lo, hi):
    """a without lo layers at the start and hi at the end of direction d."""
    return a.narrow(DIM[d], lo, a.shape[DIM[d]] - lo - hi)


class _Flow:
    def __init__(self, u, fluid, re, box=CHANNEL, open_ends=False, nut=None):
        px = pz = forcing = not open_ends
        c3, c2, c1 = u.shape[-3:]
        self.dx = (box[0] / c1, box[1] / c2, box[2] / c3)
        self.vol = self.dx[0] * self.dx[1] * self.dx[2]
        self.vis = torch.tensor([1.0 / r for r in re], dtype=F64, device=u.device).reshape(-1, 1, 1, 1)
        self.px, self.pz, self.forcing, self.nut = px, pz, forcing, nut
        self.fluid = fluid
        self.solid = _solid(fluid, px, pz)
        self.ro = torch.full_like(u[:, 0], RHO0)
        self.u = [u[:, m] for m in range(3)]
        f = [[a.contiguous() for a in t] for t in zip(*(_faces(v, fluid, px, pz) for v in u))]
        self.f = [[torch.zeros(len(a), *a[0].shape[1:], dtype=F64, device=u.device)] +
                  [torch.stack([b[m] for b in a]) for m in range(3)] for a in f]  # p, u1, u2, u3 per direction
        self.half = self.u  # the level the time step is taken from
        self.time = torch.zeros_like(self.vis)
        self.n = 0

    def cells(self, a, d):
        """a with the cell before the first and after the last along direction d."""
        n, t = a.shape[DIM[d]], DIM[d]
        lo, hi = a.narrow(t, 0, 1), a.narrow(t, n - 1, 1)
        return torch.cat((hi, a, lo) if (self.px, False, self.pz)[d] else (lo, a, hi), t)

    def ghost_faces(self, a, d):
        n, t = a.shape[DIM[d]], DIM[d]
        if (self.px, False, self.pz)[d]:
            lo, hi = a.narrow(t, n - 2, 1), a.narrow(t, 1, 1)
        else:
            lo, hi = a.narrow(t, 0, 1), a.narrow(t, n - 1, 1)
        return torch.cat((lo, a, hi), t)

    def solid_along(self, d):
        s = self.solid
        for e in range(3):
            if e != d:
                s = _cut(s, e, 1, 1)
        return s

    def stress_force(self, ro, u):
        nu = None if self.nut is None else self.nut(self, u)
        f = []
        for m in range(3):
            total = 0
            for d in range(3):
                v = self.cells(u[m], d)
                s = self.solid_along(d)
                lo, hi, sl, sh = _cut(v, d, 0, 1), _cut(v, d, 1, 0), _cut(s, d, 0, 1), _cut(s, d, 1, 0)
                vis = self.vis
                if nu is not None:
                    w = self.cells(nu, d) if d != 1 else torch.nn.functional.pad(nu, (0, 0, 1, 1))
                    vis = vis + 0.5 * (_cut(w, d, 0, 1) + _cut(w, d, 1, 0))
                sig = vis / self.dx[d] * torch.where(sl, torch.where(sh, 0.0, 2 * hi), torch.where(sh, -2 * lo, hi - lo))
                total = total + (_cut(sig, d, 1, 0) - _cut(sig, d, 0, 1)) * (self.vol / self.dx[d])
            f.append(total * ro)
        return f

    def half_step(self, ro, u, force, dt):
        flux = [0, 0, 0, 0]
        for d in range(3):
            p, *w = self.f[d]
            mass = (RHO0 + p / SOUND ** 2) * w[d]
            area = self.vol / self.dx[d]
            for q, a in enumerate([mass] + [mass * w[m] + p * (m == d) for m in range(3)]):
                flux[q] = flux[q] + (_cut(a, d, 1, 0) - _cut(a, d, 0, 1)) * area
        new = torch.where(self.fluid, ro - 0.5 * dt * flux[0] / self.vol, RHO0)
        v = []
        for m in range(3):
            a = (ro * u[m] * self.vol - 0.5 * dt * flux[m + 1]) / (new * self.vol)
            v.append(torch.where(self.fluid, a + 0.5 * dt * force[m] / (new * self.vol), 0.0))
        return new, v

    def sweep(self, d, old, new, dt):
        """The new faces normal to d from the cells before (old) and after (new) the half step."""
        a, b = (1, 0, 0)[d], (2, 2, 1)[d]
        roc = RHO0 * SOUND
        F = [self.ghost_faces(x, d) for x in self.f[d]]
        fw, bw = [_cut(x, d, 1, 0) for x in F], [_cut(x, d, 0, 1) for x in F]
        (ro0, u0), (ro1, u1) = [(self.cells(r, d), [self.cells(x, d) for x in v]) for r, v in (old, new)]
        sol = self.solid_along(d)
        n0, n1 = u0[d], u1[d]
        g0, g1 = SOUND ** 2 * (ro0 - RHO0) / roc, SOUND ** 2 * (ro1 - RHO0) / roc
        r_f, r_b, r1, r0 = fw[1 + d] + fw[0] / roc, bw[1 + d] + bw[0] / roc, n1 + g1, n0 + g0
        q_f, q_b, q1, q0 = fw[1 + d] - fw[0] / roc, bw[1 + d] - bw[0] / roc, n1 - g1, n0 - g0

        def limited(v, f, c, bk, grad):
            hi = torch.maximum(torch.maximum(f, c), bk) + dt * grad
            lo = torch.minimum(torch.minimum(f, c), bk) + dt * grad
            return torch.maximum(torch.minimum(v, hi), lo)

        dx = self.dx[d]
        r_out = limited(2 * r1 - r_b, r_f, r0, r_b, 2 * (r1 - r0) / dt + (n1 + SOUND) * (r_f - r_b) / dx)
        q_src = (q1 - q0) if d == 1 else (r1 - r0)
        q_out = limited(2 * q1 - q_f, q_f, q0, q_b, 2 * q_src / dt + (n1 - SOUND) * (q_f - q_b) / dx)
        tang = []
        for m in (a, b):
            tf, tb, t1, t0 = fw[1 + m], bw[1 + m], u1[m], u0[m]
            grad = 2 * (t1 - t0) / dt + n1 * (tf - tb) / dx
            tang.append([limited(2 * t1 - tb, tf, t0, tb, grad), limited(2 * t1 - tf, tf, t0, tb, grad)])
        if d == 0 and not self.px:  # inflow and outflow of a bounded x
            r_out[..., 0] = (~sol[..., 1]).to(F64)
            q_out[..., -1] = 5.0 / 6.0
            for t in tang:
                t[0][..., 0] = 0.0
                t[1][..., -1] = 0.0
        behind, ahead = lambda x: _cut(x, d, 0, 1), lambda x: _cut(x, d, 1, 0)
        sb, sf, ub, uf = behind(sol), ahead(sol), behind(n1), ahead(n1)
        r, q = behind(r_out), ahead(q_out)
        open_, wall_b, wall_f = ~sb & ~sf, sb & ~sf, ~sb & sf
        from_b = ((uf >= 0) & (ub >= 0)) | ((ub >= 0) & (uf <= 0) & ~((uf <= 0) & (ub <= 0)) & (ub > -uf))
        from_f = ((uf <= 0) & (ub <= 0)) | ((ub >= 0) & (uf <= 0) & (ub <= -uf))
        in_f, in_b = uf <= 0, ub >= 0  # towards the wall: extrapolated; away from it: the cell's own values
        c2 = SOUND ** 2
        p = torch.where(open_, 0.5 * (r - q) * roc,
                        torch.where(wall_b, torch.where(in_f, -q * roc, (ahead(ro1) - RHO0) * c2),
                                    torch.where(wall_f, torch.where(in_b, r * roc, (behind(ro1) - RHO0) * c2), 0.0)))
        out = [p, None, None, None]
        out[1 + d] = torch.where(open_, 0.5 * (r + q), 0.0)
        for m, t in ((a, tang[0]), (b, tang[1])):
            mid = ahead(u1[m]) + behind(u1[m]) - self.f[d][1 + m]
            own_f, own_b = (uf, ub) if d == 1 and m == a else (ahead(u1[m]), behind(u1[m]))
            tb, tf = behind(t[0]), ahead(t[1])
            out[1 + m] = torch.where(open_, torch.where(from_b, tb, torch.where(from_f, tf, mid)),
                                     torch.where(wall_b, torch.where(in_f, tf, own_f),
                                                 torch.where(wall_f, torch.where(in_b, tb, own_b), 0.0)))
        return out

    def step(self):
        top = lambda a: a.abs().amax((-3, -2, -1), keepdim=True)
        dts = [CFL * self.dx[d] / (SOUND + top(self.half[d])) for d in range(3)]
        dts += [CFL * h * h / (2 * self.vis) for h in self.dx]
        dt = dts[0]
        for v in dts[1:]:
            dt = torch.minimum(dt, v)
        fl = self.fluid
        self.ub, self.g = torch.zeros_like(dt), torch.zeros_like(dt)
        force = self.stress_force(self.ro, self.u)
        if self.forcing:
            self.ub = (self.u[0] * fl).sum((-3, -2, -1), keepdim=True) / fl.sum()
            self.g = (1.0 - self.ub) / dt
            force[0] = force[0] + self.ro * self.vol * self.g
        force = [f * fl for f in force]
        new = self.half_step(self.ro, self.u, force, dt)
        self.f = [self.sweep(d, (self.ro, self.u), new, dt) for d in range(3)]
        self.half = new[1]
        self.ro, self.u = self.half_step(*new, force, dt)
        self.dt, self.time, self.n = dt, self.time + dt, self.n + 1

    def field(self, name):
        if name in CELLS:
            return self.ro if name == "ronCon" else self.u[int(name[1]) - 1]
        return self.f[int(name[-1]) - 1][0 if name[0] == "p" else int(name[1])]


def _gradient(flow, u):
    """d u_m / d x_d by central differences; a solid neighbour counts as minus the cell."""
    A = []
    for m in range(3):
        row = []
        for d in range(3):
            v, s = flow.cells(u[m], d), flow.solid_along(d)
            hi = torch.where(_cut(s, d, 2, 0), -u[m], _cut(v, d, 2, 0))
            lo = torch.where(_cut(s, d, 0, 2), -u[m], _cut(v, d, 0, 2))
            row.append((hi - lo) / (2 * flow.dx[d]))
        A.append(torch.stack(row, -1))
    return torch.stack(A, -2)


def _features(A, c2, scale):
    """The ten invariants of velocity gradients A [..., k, j, i, 3, 3]."""
    T = A.transpose(-1, -2)
    S, W = 0.5 * (A + T), 0.5 * (A - T)
    tr = lambda M: M.diagonal(dim1=-2, dim2=-1).sum(-1)
    root = lambda x, n: x.sign() * x.abs() ** (1.0 / n)
    y = _heights(c2)[:, None]
    S2, W2 = S @ S, W @ W
    f = [tr(S), tr(S2).clamp(min=0).sqrt(), (-tr(W2)).clamp(min=0).sqrt(), root(tr(S2 @ S), 3), root(tr(W2 @ S), 3),
         root(tr(W2 @ S2), 4), root(tr(W2 @ S @ W @ S2), 6), -y.sign() * S[..., 0, 1], -y.sign() * W[..., 0, 1]]
    f.append(((0.5 * CHANNEL[1] - y.abs()) * scale).expand_as(f[0]))
    return torch.stack(f, -1)


def _layers(w):
    return w[:320].reshape(32, 10), w[320:352], w[352:1376].reshape(32, 32), w[1376:1408], w[1408:1440], w[1440]


def _forward(w, x):
    w1, b1, w2, b2, w3, b3 = _layers(w)
    gelu = lambda z: torch.nn.functional.gelu(z, approximate="tanh")
    return torch.nn.functional.softplus(gelu(gelu(x @ w1.T + b1) @ w2.T + b2) @ w3 + b3)


def _eddy_viscosity(seed):
    w, mu, sd = (torch.from_numpy(a).to(_dev()) for a in _network(seed))
    w = w.to(torch.bfloat16).to(F64)

    def nut(flow, u):
        x = _features(_gradient(flow, u), u[0].shape[-2], U_TAU / flow.vis.reshape(-1)[0])
        return _forward(w, (x - mu) / sd) * flow.vis

    return nut


def _exact_train(case, seed):
    x, t = (a.to(F64) for a in _rows(case, seed))
    mu, sd = x.mean(0), x.std(0, correction=0)
    x = (x - mu) / sd
    w = torch.from_numpy(_network(seed)[0]).to(_dev())
    m, v = torch.zeros_like(w), torch.zeros_like(w)
    batches, loss = case["rows"] // case["batch"], 0.0
    for b in range(batches):
        at = torch.arange(case["batch"], device=x.device) * batches + b
        q = w.to(torch.bfloat16).to(F64).requires_grad_()
        e = ((_forward(q, x[at]) - t[at]) ** 2).mean()
        g, = torch.autograd.grad(e, q)
        loss += float(e) / batches
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        w = w - 1e-3 * (m / (1 - 0.9 ** (b + 1))) / ((v / (1 - 0.999 ** (b + 1))).sqrt() + 1e-8)
    return {"loss": loss, "weights": w}


def _exact_samples(case, seed):
    size = (case["c1"], case["c2"], case["c3"])
    u = _velocity(seed, *size, 0.1, False)
    if not case["fp64"]:
        u = u.float().to(F64)
    flow = _Flow(u[None], _fluid(*size, False), [5600.0])

    def box(a, sign):
        for d in range(3):
            v = flow.cells(a, d)
            lo, hi = _cut(v, d, 0, 2), _cut(v, d, 2, 0)
            if d == 1:
                lo, hi = lo.clone(), hi.clone()
                lo[..., 0, :], hi[..., -1, :] = sign * a[..., 0, :], sign * a[..., -1, :]
            a = (lo + a + hi) / 3
        return a

    U = [u[None, m] for m in range(3)]
    F = [box(a, -1.0) for a in U]
    s = case["stride"]
    pick = lambda a: a[0, ::s, :, ::s]
    A = pick(_gradient(flow, F))
    x = _features(A, size[1], U_TAU * 5600.0)
    tau = torch.stack([torch.stack([pick(box(U[a] * U[b], 1.0) - F[a] * F[b]) for b in range(3)], -1) for a in range(3)], -2)
    eye = torch.eye(3, dtype=F64, device=u.device)
    dev = lambda M: M - M.diagonal(dim1=-2, dim2=-1).sum(-1)[..., None, None] / 3 * eye
    S, T = dev(0.5 * (A + A.transpose(-1, -2))), dev(tau)
    num, den = -(T * S).sum((-2, -1)), 2 * (S * S).sum((-2, -1))
    t = torch.where(den > 1e-30, (num / den).clamp(min=0), 0.0) * 5600.0
    return {"features": x.reshape(-1, 10), "targets": t.reshape(-1)}


def _exact_statistics(case, seed):
    size = (case["c1"], case["c2"], case["c3"])
    u = _velocity(seed, *size, 0.1, False)
    if not case["fp64"]:
        u = u.float().to(F64)
    prof = u[0].mean((0, 2))
    dy = CHANNEL[1] / size[1]
    pairs = [u[0], u[1], u[2], u[0] ** 2, u[1] ** 2, u[2] ** 2, u[0] * u[1], u[0] * u[2], u[1] * u[2]]
    kin = float((u ** 2).sum() / 2)
    n = u[0].numel()
    return {"profile": prof, "shear": 2 / 5600.0 * prof[[0, -1]] / dy, "planes": torch.stack([a.mean((0, 2)) for a in pairs], -1),
            "energy": kin * math.prod(CHANNEL), "sums": [RHO0 * n] + [float(u[m].sum()) * RHO0 for m in range(3)] + [kin], "cells": n}


def exact(case, seed):
    if not torch.cuda.is_available():
        return None
    kind = case["kind"]
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "samples":
        return _exact_samples(case, seed)
    if kind == "statistics":
        return _exact_statistics(case, seed)
    if kind == "ensemble":
        members, out = _ensemble_members(case, seed), {}
        for c in sorted({m[0] for m in members}):
            of = [m for m in members if m[0] == c]
            flow = _Flow(torch.stack([_velocity(m[3], *c, m[2], False) for m in of]), _fluid(*c, False), [m[1] for m in of])
            for _ in range(case["steps"]):
                flow.step()
            out[f"{c[0]}x{c[1]}x{c[2]}"] = {n: flow.field(n) for n in CELLS}
        return out
    if case["c1"] * case["c2"] * case["c3"] * case["steps"] > 4e9:
        return None  # over about 20 seconds
    step, open_ends = case.get("step", False), bool(case.get("step") or case.get("bounded"))
    size = (case["c1"], case["c2"], case["c3"])
    flow = _Flow(_velocity(seed, *size, 0.01 if step else 0.1, step)[None], _fluid(*size, step), [case["re"]], _box(case),
                 open_ends, _eddy_viscosity(seed) if case.get("closure") else None)
    for _ in range(case["steps"]):
        flow.step()
    return {"scalars": {"dt": float(flow.dt), "time": float(flow.time), "nstep": flow.n, "ub": float(flow.ub), "g": float(flow.g)},
            "fields": {n: flow.field(n)[0] for n in CELLS + FACES}}
