"""The calls this framework is timed on, through its public entry points: `Sim` (steps, ionization,
the FUV field, the stirring phase, the renderer's voxel pack, snapshots) and `BatchSim`.

Scenes are the package's own synthetic initial conditions (nebulaviewer_gb300.ics) at sizes between
the smallest preview grid and a grid of 134 million cells.  Launch shapes are the library's defaults.
`exact` restates the scheme in float64 torch, without this package's kernels.

A case's `kind`:
  step      Sim.step(k): a simulation loop (viewer, bake), blocking as the API is
  ionize    Sim.ionize(): a star or a live parameter changed
  fuv       Sim.fuv_field(): the FUV field of a frame
  stir      Sim.step(k) in the stirring phase
  frame     the viewer's frame: Sim.step(k), Sim.update_render_fields(), Sim.render_pack()
  render    Sim.render_pack() alone: a look parameter changed
  snapshot  Sim.snapshot_pack() and Sim.snapshot_unpack(): the timeline's capture and restore
  batch     BatchSim.step(k) over instances of different sizes
A run that has stepped `restart` steps starts over from its first state, as a program that replays a
scene does, so the gas stays the scene's.
"""
import math
import random

import numpy as np
import torch

from nebulaviewer_gb300 import ics, stir
from nebulaviewer_gb300.batch import BatchSim
from nebulaviewer_gb300.params import make_params, sound_speeds
from nebulaviewer_gb300.sim import Sim

LOOK = {"c_ha": (0.33, 0.675, 1.5), "c_o3": (0.45, 1.125, 1.5), "c_s2": (1.2, 0.66, 0.3), "c_dg": (0.07, 0.035, 0.01),
        "c_sh": (0.02, 0.007, 0.009), "gs": 12.0, "ambient": 0.1, "edge": 0.08}

BASE = dict(scene="sheet", nx=64, ny=64, nz=64, stars=1, steps=1, solver="hll", limiter="minmod", arith="fast",
            fp32_fields=False, jets=False, restart=240)


def _case(name, kind, **kw):
    return {"name": name, "kind": kind, **BASE, **kw}


def listed():
    return [
        # the plain 64^3 torus with one star, one step a call: launches and the blocking read count
        _case("step_torus_64", "step", scene="torus"),
        # the headline workload: the 256^3 sheet with six stars and wind, one ionization and three steps
        _case("step_sheet_256", "step", nx=256, ny=256, nz=256, stars=6, steps=3),
        # a large grid with the plane-parallel source: the cloud wall, 134 M cells
        _case("step_wall_512", "step", scene="cliffwall", nx=512, ny=512, nz=512, stars=3, steps=3),
        # a cropped slab of odd sizes, jets on, van Leer, float32 front and FUV fields
        _case("step_slab_ragged", "step", nx=97, ny=161, nz=228, stars=4, steps=3, limiter="vanleer", jets=True,
              fp32_fields=True),
        # the bit-exact build, as a parity run uses it
        _case("step_exact_128", "step", nx=128, ny=128, nz=128, stars=6, steps=3, arith="exact"),
        # the first-order-safe solver on a mid-size grid (a quick preview of a cloud wall)
        _case("step_rusanov_160", "step", scene="cliffwall", nx=160, ny=160, nz=160, stars=3, steps=3, solver="rusanov"),
        # a star's photon rate was changed: ionize at once
        _case("ionize_sheet_192", "ionize", nx=192, ny=192, nz=192, stars=6),
        # a frame's FUV field with the 256^3 grid's ray budget
        _case("fuv_sheet_256", "fuv", nx=256, ny=256, nz=256, stars=6),
        # turbulence before the stars switch on
        _case("stir_torus_192", "stir", scene="torus", nx=192, ny=192, nz=192, steps=4),
        # the interactive viewer's loop on a preview grid
        _case("frame_torus_96", "frame", scene="torus", nx=96, ny=96, nz=96, stars=2, steps=4),
        # the look was changed, or the timeline captures and restores
        _case("snapshot_sheet_256", "snapshot", nx=256, ny=256, nz=256, stars=6),
        # eight instances of 64^3 to 192^3 and a slab, stepped together
        _case("batch_8", "batch", scene="mixed", nx=64, ny=64, nz=192, instances=8, steps=3),
    ]


def _size(rng, lo, hi, mult=1):
    return max(mult, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / mult)) * mult)


def draw(rng):
    kind = rng.choice(["step", "step", "step", "ionize", "fuv", "stir", "frame", "render", "snapshot", "batch"])
    c = dict(BASE, kind=kind)
    top = 320 if kind == "step" else 256
    if rng.random() < 0.4:
        c["nx"] = c["ny"] = c["nz"] = _size(rng, 48, top, 4)
    else:
        c["nx"], c["ny"], c["nz"] = _size(rng, 40, top), _size(rng, 40, top), _size(rng, 40, top, 4)
    c["scene"] = rng.choice(["torus", "sheet", "sheet", "cliffwall"])
    c["stars"] = 3 if c["scene"] == "cliffwall" else rng.randint(1, 8)
    c["steps"] = rng.choice([1, 2, 3, 4, 6])
    c["fp32_fields"] = rng.random() < 0.2
    if kind == "step":
        c["solver"] = rng.choice(["hll", "hll", "hll", "rusanov"])
        c["limiter"] = rng.choice(["minmod", "minmod", "vanleer", "mc"])
        c["arith"] = rng.choice(["fast", "fast", "fast", "exact"])
        c["jets"] = rng.random() < 0.3
    elif kind == "stir":
        c["scene"], c["stars"] = "torus", 1
    elif kind == "batch":
        c.update(scene="mixed", nx=48, ny=48, nz=rng.choice([96, 128, 160, 192]), instances=rng.randint(2, 8),
                 fp32_fields=False)
    return c


# ------------------------------------------------------------------ inputs
def _instances(case):
    """(shape, scene, stars) of a batch: cubes with edges between nx and nz, every fourth a cropped
    slab, as ics.batch_scenes mixes them"""
    rng = random.Random(1000 * case["instances"] + case["nz"])
    slabs, out = [(96, 160, 288), (160, 96, 224), (128, 192, 96)], []
    for m in range(case["instances"]):
        e = 8 * rng.randint(case["nx"] // 8, case["nz"] // 8)
        shape = slabs[(m // 4) % 3] if m % 4 == 3 else (e, e, e)
        out.append((shape, rng.choice(["torus", "sheet"]), rng.randint(1, 8)))
    return out


def _scenes(case, seed, device):
    """the initial conditions of a case: a list of dicts as nebulaviewer_gb300.ics makes them"""
    if case["kind"] == "batch":
        out = []
        for m, (shape, scene, stars) in enumerate(_instances(case)):
            gen = ics.torus if scene == "torus" else ics.sheet
            kw = {} if scene == "torus" else {"res": min(shape)}
            out.append(gen(seed=seed + m, device=device, shape=shape, nstars=stars, **kw))
        return out
    shape = (case["nx"], case["ny"], case["nz"])
    if case["kind"] == "stir":
        ic = ics.torus(seed=seed, device=device, shape=shape, stir=True)
        # the forcing of the scene, renewed less often than a run starts over: the list of fields never ends
        ic["P"].update(pre_t=1e6, pre_corr=2.0, drive_main=0.0)
        grid = stir.forcing_grid([n * ic["dx"] for n in shape], ic["dx"], shape)
        rng = np.random.default_rng(seed)
        ic["stir_grid"] = grid
        ic["stir_fields"] = [np.stack(stir.solenoidal(grid[0], rng, 1.0, 4.0)) for _ in range(4)]
    elif case["scene"] == "torus":
        ic = ics.torus(seed=seed, device=device, shape=shape, nstars=case["stars"])
    elif case["scene"] == "sheet":
        ic = ics.sheet(res=min(shape), seed=seed, nstars=case["stars"], device=device, shape=shape)
    else:
        ic = ics.cliffwall(res=min(shape), seed=seed, device=device, shape=shape)
    ic["P"].update(solver=case["solver"], limiter=case["limiter"])
    if case["fp32_fields"]:
        ic["P"]["fp32_fields"] = True
    if case["jets"]:
        n = len(ic["stars"])
        ax = np.random.default_rng(seed + 7).standard_normal((n, 3))
        ax /= np.linalg.norm(ax, axis=1, keepdims=True)
        ic["jets"] = [tuple(float(v) for v in a) for a in ax]
        ic["jkinds"] = ["jet" if s % 2 == 0 else "none" for s in range(n)]
        ic["P"].update(jet=3000.0, jet_angle=25.0, jet_r=0.08)
    return [ic]


class State:
    """a program's simulation(s) and the first state it goes back to"""

    def __init__(self, case, seed):
        self.case = case
        self.sims = []
        for ic in _scenes(case, seed, "cuda"):
            self.sims.append(Sim.from_state(ic["shape"], ic["dx"], ic["rho"], ic["stars"], ic["kinds"], ic["jets"],
                                            ic["jkinds"], ic["P"], mom=ic["mom"], torus=ic.get("torus"),
                                            stir_fields=ic.get("stir_fields"), stir_grid=ic.get("stir_grid"),
                                            arith=case["arith"], device="cuda:0"))
        self.sim = self.sims[0]
        self.done, self.fresh = 0, True
        self.look = dict(LOOK, inv_L=[1.0 / v for v in self.sim.L], dx=self.sim.dx)
        if case["kind"] in ("render", "snapshot"):
            self.sim.update_render_fields(force=True)
        if case["kind"] == "snapshot":
            n = case["nx"] * case["ny"] * case["nz"]
            self.buf = torch.empty(13 * n, dtype=torch.uint8, device="cuda")
        self.first = None
        if case["kind"] in ("step", "stir", "frame", "batch"):
            self.first = [(s.get_state_meta(), [t.clone() for t in _fields(s)]) for s in self.sims]
        self.batch = BatchSim(self.sims) if case["kind"] == "batch" else None

    def advance(self, k):
        if self.done + k > self.case["restart"]:
            for s, (meta, saved) in zip(self.sims, self.first):
                for t, v in zip(_fields(s), saved):
                    t.copy_(v)
                s.set_state_meta(meta)
            self.done, self.fresh = 0, True
        (self.batch or self.sim).step(k)
        self.done += k


def _fields(s):
    return [f.torch() for f in (s.rho, s.mx, s.my, s.mz, s.xi, s.dfront, s.g0)]


def prepare(case, seed):
    return State(case, seed)


def run(state):
    kind, sim, k = state.case["kind"], state.sim, state.case["steps"]
    if kind in ("step", "stir"):
        state.advance(k)
        return dict(zip(("rho", "mx", "my", "mz", "xi", "dfront"), _fields(sim)))
    if kind == "batch":
        state.advance(k)
        return [dict(zip(("rho", "mx", "my", "mz", "xi", "dfront"), _fields(s))) for s in state.sims]
    if kind == "ionize":
        sim.ionize()
        return {"xi": sim.xi.torch(), "dfront": sim.dfront.torch()}
    if kind == "fuv":
        sim.fuv_field()
        return {"g0": sim.g0.torch()}
    if kind == "frame":
        state.advance(k)
        sim.update_render_fields(force=state.fresh)
        state.fresh = False
        return {"voxels": sim.render_pack(state.look).torch(), "g0": sim.g0.torch(), "rho": sim.rho.torch()}
    if kind == "render":
        return {"voxels": sim.render_pack(state.look).torch()}
    sim.snapshot_pack(state.buf)
    sim.snapshot_unpack(state.buf)
    return {"snapshot": state.buf, "rho": sim.rho.torch(), "xi": sim.xi.torch()}


# ------------------------------------------------------------------ what a pass cannot do without
def _ray_budget(nz):
    nu = 512 if nz <= 256 else 1024
    fuv = (128, 128, 256) if nz <= 192 else ((160, 160, 320) if nz <= 256 else (256, 256, 512))
    return nu, 2 * nu, fuv


def _cells(case):
    if case["kind"] != "batch":
        return case["nx"] * case["ny"] * case["nz"]
    return sum(a * b * c for (a, b, c), _, _ in _instances(case))


def work(case):
    """bytes: a step reads rho, m, xi and writes rho, m (36 B / cell); an ionization reads rho and
    writes xi and the front distance; the FUV field reads rho, xi and writes G0; stirring is folded
    into the step; voxels and snapshots read their fields and write their bytes.  flops: two RK2
    stages of three reconstructed face fluxes a cell."""
    n, k = _cells(case), case["steps"]
    h = 4 if case["fp32_fields"] else 2
    nu, nphi, _ = _ray_budget(case["nz"])
    kind = case["kind"]
    ion, fuv, vox = (8 + h) * n, (8 + h) * n, (20 + 2 * h + 8) * n
    if kind in ("step", "batch"):
        return {"bytes": 36 * n * k + ion * -(-k // 3), "flops": 660.0 * n * k}
    if kind == "stir":
        return {"bytes": 36 * n * k, "flops": 660.0 * n * k}
    if kind == "ionize":
        return {"bytes": ion, "flops": 40.0 * n * case["stars"]}
    if kind == "fuv":
        return {"bytes": fuv, "flops": 60.0 * n * case["stars"]}
    if kind == "frame":
        return {"bytes": 36 * n * k + ion * -(-k // 3) + fuv / 2 + vox, "flops": 660.0 * n * k}
    if kind == "render":
        return {"bytes": vox, "flops": 100.0 * n}
    # pack: every field in, 13 B out; unpack: 13 B in, every field out
    return {"bytes": 2 * (20 + 2 * h + 13) * n, "flops": 20.0 * n}


# ------------------------------------------------------------------ float64 restatement
def _minmod(a, b):
    return torch.where(a * b <= 0, torch.zeros_like(a), torch.where(a.abs() < b.abs(), a, b))


def _vanleer(a, b):
    return torch.where(a * b <= 0, torch.zeros_like(a), 2.0 * a * b / (a + b))


def _mc(a, b):
    s = torch.sign(a) * torch.minimum(torch.minimum(2.0 * a.abs(), 2.0 * b.abs()), 0.5 * (a + b).abs())
    return torch.where(a * b <= 0, torch.zeros_like(a), s)


def _edge_pad(a, ax, w):
    lo, hi = a.narrow(ax, 0, 1), a.narrow(ax, a.shape[ax] - 1, 1)
    return torch.cat([lo] * w + [a] + [hi] * w, dim=ax)


class Exact:
    """the scheme of the simulation step in float64 torch"""

    def __init__(self, ic):
        self.P = P = make_params(base=ic["P"])
        self.cn2, self.ci2, self.vmax = sound_speeds(P)
        self.shape, self.dx = tuple(ic["shape"]), float(ic["dx"])
        self.dev = ic["rho"].device
        f64 = dict(device=self.dev, dtype=torch.float64)
        self.U = [ic["rho"].to(torch.float32).double()]
        self.U += [torch.zeros(self.shape, **f64) for _ in range(3)] if ic["mom"] is None else \
            [v.to(torch.float32).double() for v in ic["mom"]]
        self.xi = torch.zeros(self.shape, **f64)
        self.df = torch.full(self.shape, 1e3, **f64)
        self.g0 = torch.zeros(self.shape, **f64)
        self.stars, self.jets, self.jkinds = ic["stars"], ic["jets"], ic["jkinds"]
        self.t, self.it, self.clock = 0.0, 0, 0.0
        self.L = [n * self.dx for n in self.shape]
        self.diag = math.sqrt(sum(v * v for v in self.L)) + 0.6
        self.nsteps = int(self.diag / self.dx) + 1               # the fast ray budget: one sample per cell
        self.axis = [((torch.arange(n, **f64) + 0.5) * self.dx).reshape([-1 if a == d else 1 for d in range(3)])
                     for a, n in enumerate(self.shape)]

    # ---- hydro
    def max_speed(self):
        r, mx, my, mz = self.U
        c = torch.sqrt(self.cn2 + self.xi * (self.ci2 - self.cn2))
        return float(((mx.abs() + my.abs() + mz.abs()) / r + c).max())

    def flux_diff(self, q, c2, c, ax):
        """F(+1/2) - F(-1/2) of the four conserved components along `ax`"""
        floor, n = float(self.P["floor"]), self.shape[ax]
        lim = {"minmod": _minmod, "vanleer": _vanleer, "mc": _mc}[self.P["limiter"]]
        rus = self.P["solver"] == "rusanov"
        lim = _minmod if rus else lim
        L, R = [], []
        for v in q:
            v = _edge_pad(v, ax, 2)
            d = v.narrow(ax, 1, n + 3) - v.narrow(ax, 0, n + 3)
            s = 0.5 * lim(d.narrow(ax, 0, n + 2), d.narrow(ax, 1, n + 2))
            L.append(v.narrow(ax, 1, n + 1) + s.narrow(ax, 0, n + 1))
            R.append(v.narrow(ax, 2, n + 1) - s.narrow(ax, 1, n + 1))
        del d, s
        c2, c = _edge_pad(c2, ax, 1), _edge_pad(c, ax, 1)
        c2L, c2R, cL, cR = c2.narrow(ax, 0, n + 1), c2.narrow(ax, 1, n + 1), c.narrow(ax, 0, n + 1), c.narrow(ax, 1, n + 1)
        rL, rR = L[0].clamp_min(floor), R[0].clamp_min(floor)
        uL, uR = L[1 + ax], R[1 + ax]
        one = torch.ones_like(rL)
        if rus:
            ha = 0.5 * torch.maximum(uL.abs() + cL, uR.abs() + cR)
        else:
            SL = torch.minimum(uL - cL, uR - cR).clamp_max(0.0)
            SR = torch.maximum(uL + cL, uR + cR).clamp_min(0.0)
        out = []
        for k in range(4):
            UL, UR = rL * (one if k == 0 else L[k]), rR * (one if k == 0 else R[k])
            FL, FR = UL * uL, UR * uR
            if k == 1 + ax:
                FL, FR = FL + rL * c2L, FR + rR * c2R
            F = 0.5 * (FL + FR) - ha * (UR - UL) if rus else (SR * FL - SL * FR + SL * SR * (UR - UL)) / (SR - SL)
            out.append(F.narrow(ax, 1, n) - F.narrow(ax, 0, n))
        return out

    def stage(self, U, U0, a, b, dt, pulse, sources):
        P, floor = self.P, float(self.P["floor"])
        r = U[0].clamp_min(floor)
        q = [r] + [m / r for m in U[1:]]
        c2 = self.cn2 + self.xi * (self.ci2 - self.cn2)
        c = torch.sqrt(c2)
        dU = [torch.zeros_like(r) for _ in range(4)]
        for ax in range(3):
            for k, d in enumerate(self.flux_diff(q, c2, c, ax)):
                dU[k] -= d / self.dx
        del q
        X = self.axis
        if sources and float(P["wind"]) > 0.0:
            w = float(P["wind"]) * self.xi * U[0] * (self.xi > 0.01)
            for s in self.stars:
                R = [x - float(np.float32(p)) for x, p in zip(X, s[:3])]
                r2 = R[0] ** 2 + R[1] ** 2 + R[2] ** 2 + 0.0004
                f = w * s[3] / (r2 * torch.sqrt(r2))
                for k in range(3):
                    dU[1 + k] += f * R[k]
        if sources and float(P["jet"]) > 0.0:
            cut = math.cos(math.radians(float(P["jet_angle"])))
            for s, j, kind in zip(self.stars, self.jets, self.jkinds):
                if kind != "jet":
                    continue
                R = [x - float(np.float32(p)) for x, p in zip(X, s[:3])]
                rr = torch.sqrt(R[0] ** 2 + R[1] ** 2 + R[2] ** 2)
                cth = (R[0] * j[0] + R[1] * j[1] + R[2] * j[2]) / rr.clamp_min(1e-12)
                on = (rr < float(P["jet_r"])) & (rr > 1e-6) & (cth.abs() > cut)
                f = torch.where(on, torch.where(cth > 0, 1.0, -1.0) * float(P["jet"]) * pulse / (rr * rr + 0.0004), 0.0)
                for k in range(3):
                    dU[1 + k] += U[0] * j[k] * f
        o = [a * u0 + b * (u + dt * d) for u0, u, d in zip(U0, U, dU)]
        r = o[0].clamp_min(floor)
        v = [m / r for m in o[1:]]
        sp = torch.sqrt(v[0] ** 2 + v[1] ** 2 + v[2] ** 2)
        f = torch.where(sp > self.vmax, self.vmax / sp.clamp_min(1e-300), 1.0)
        return [r] + [r * vk * f for vk in v]

    def step(self, ion_every):
        if self.it % ion_every == 0:
            self.ionize()
        P = self.P
        dt = float(P["cfl"]) * self.dx / self.max_speed()
        pulse = max(0.0, 1.0 + float(P["jet_pulse"]) * math.sin(2.0 * math.pi * self.t / float(P["jet_period"])))
        U1 = self.stage(self.U, self.U, 0.0, 1.0, dt, pulse, True)
        self.U = self.stage(U1, self.U, 0.5, 0.5, dt, pulse, True)
        self.t += dt
        self.it += 1

    def pre_step(self, A, B, dxs):
        P = self.P
        dt = float(P["cfl"]) * self.dx / self.max_speed()
        U1 = self.stage(self.U, self.U, 0.0, 1.0, dt, 1.0, False)
        self.U = self.stage(U1, self.U, 0.5, 0.5, dt, 1.0, False)
        blend = min(self.clock / float(P["pre_corr"]), 1.0)
        n = A.shape[1:]
        ix = []
        for x, m in zip(self.axis, n):
            g = x.reshape(-1) / dxs - 0.5
            out = (g < -0.5) | (g > m - 0.5)
            i = torch.floor(g).long()
            ix.append((i.clamp(0, m - 1), (i + 1).clamp(0, m - 1), g - i, ~out))
        inside = ix[0][3][:, None, None] & ix[1][3][None, :, None] & ix[2][3][None, None, :]
        for k in range(3):
            f = (1.0 - blend) * A[k] + blend * B[k]
            for ax in range(3):
                i0, i1, w, _ = ix[ax]
                w = w.reshape([-1 if a == ax else 1 for a in range(3)])
                f = f.index_select(ax, i0) * (1.0 - w) + f.index_select(ax, i1) * w
            self.U[1 + k] = self.U[1 + k] + self.U[0] * float(P["pre_amp"]) * dt * f * inside
        self.clock += dt

    # ---- rays
    def _dirs(self, nu, nphi):
        f64 = dict(device=self.dev, dtype=torch.float64)
        u = -1.0 + (torch.arange(nu, **f64) + 0.5) * 2.0 / nu
        s = torch.sqrt((1.0 - u * u).clamp_min(0.0))
        phi = (torch.arange(nphi, **f64) + 0.5) * 2.0 * math.pi / nphi
        return torch.stack([(s[:, None] * torch.cos(phi)).reshape(-1), (s[:, None] * torch.sin(phi)).reshape(-1),
                            u[:, None].expand(nu, nphi).reshape(-1)])

    def _range(self, o, d):
        t0, t1 = torch.zeros_like(d[0]), torch.full_like(d[0], 1e9)
        for a in range(3):
            ta, tb = -o[a] / d[a], (self.L[a] - o[a]) / d[a]
            t0, t1 = torch.maximum(t0, torch.minimum(ta, tb)), torch.minimum(t1, torch.maximum(ta, tb))
        n0 = (t0 / self.dx).long()
        return n0, torch.clamp((t1.clamp_max(1e6) / self.dx).long() + 2, max=self.nsteps)

    def _sample(self, fields, p):
        nx, ny, nz = self.shape
        idx, fr, out = [], [], None
        for x, n in zip(p, self.shape):
            g = x / self.dx - 0.5
            bad = (g < -0.5) | (g > n - 0.5)
            out = bad if out is None else out | bad
            i = torch.floor(g).long()
            idx.append((i.clamp(0, n - 1), (i + 1).clamp(0, n - 1)))
            fr.append(g - i)
        res = [0.0] * len(fields)
        for a in range(2):
            for b in range(2):
                ij = (idx[0][a] * ny + idx[1][b]) * nz
                wab = (fr[0] if a else 1.0 - fr[0]) * (fr[1] if b else 1.0 - fr[1])
                for e in range(2):
                    w = wab * (fr[2] if e else 1.0 - fr[2])
                    q = ij + idx[2][e]
                    res = [v + w * f.reshape(-1)[q] for v, f in zip(res, fields)]
        return [torch.where(out, 0.0, v) for v in res]

    def _fronts(self, star, nu, nphi):
        o = [float(np.float32(v)) for v in star[:3]]
        Q = star[3] * float(self.P["q_main"])
        d = self._dirs(nu, nphi)
        rf = torch.full_like(d[0], self.diag)
        n, n1 = self._range(o, d)
        col = torch.zeros_like(rf)
        live = torch.nonzero(n < n1).reshape(-1)
        d, n, n1, col = d[:, live], n[live], n1[live], col[live]
        while live.numel():
            r = (n + 0.5) * self.dx
            nv, = self._sample([self.U[0]], [o[a] + d[a] * r for a in range(3)])
            inc = nv * nv * r * r * self.dx
            cross = col + inc > Q
            rf[live[cross]] = (r - 0.5 * self.dx + self.dx * (Q - col) / inc.clamp_min(1e-20))[cross]
            col, n = col + inc, n + 1
            keep = ~cross & (n < n1)
            live, d, n, n1, col = live[keep], d[:, keep], n[keep], n1[keep], col[keep]
        return rf.reshape(nu, nphi)

    def _polar(self, star):
        o = [float(np.float32(v)) for v in star[:3]]
        R = [x - p for x, p in zip(self.axis, o)]
        r = torch.sqrt(R[0] ** 2 + R[1] ** 2 + R[2] ** 2).clamp_min(1e-6)
        phi = torch.atan2(R[1], R[0])
        phi = torch.where(phi < 0, phi + 2.0 * math.pi, phi).expand(self.shape)
        return r, R[2] / r, phi

    @staticmethod
    def _lin(g, n, wrap):
        i = torch.floor(g).long()
        ends = (i % n, (i + 1) % n) if wrap else (i.clamp(0, n - 1), (i + 1).clamp(0, n - 1))
        return ends, g - i

    def ionize(self):
        nu, nphi, _ = _ray_budget(self.shape[2])
        xi, df, width = torch.zeros_like(self.xi), torch.full_like(self.df, 1e3), 1.2 * self.dx
        for s in self.stars:
            tab = self._fronts(s, nu, nphi).reshape(-1)
            for sl in range(0, self.shape[0], 64):               # slabs: the index arrays are large
                r, u, phi = (v[sl:sl + 64] for v in self._polar(s))
                (u0, u1), tu = self._lin((u + 1.0) * 0.5 * nu - 0.5, nu, False)
                (p0, p1), tp = self._lin(phi / (2.0 * math.pi) * nphi - 0.5, nphi, True)
                ra = tab[u0 * nphi + p0] * (1.0 - tp) + tab[u0 * nphi + p1] * tp
                rb = tab[u1 * nphi + p0] * (1.0 - tp) + tab[u1 * nphi + p1] * tp
                rf = ra * (1.0 - tu) + rb * tu
                xi[sl:sl + 64] = torch.maximum(xi[sl:sl + 64], ((rf - r) / width + 0.5).clamp(0.0, 1.0))
                df[sl:sl + 64] = torch.minimum(df[sl:sl + 64], r - rf)
        F = float(self.P.get("plane_flux", 0.0) or 0.0)
        if F > 0.0:
            inc = self.U[0] ** 2 * self.dx
            col = torch.cumsum(inc, 0)
            hit = col > F
            i = hit.to(torch.uint8).argmax(0, keepdim=True)
            at = inc.gather(0, i)
            xf = i * self.dx + self.dx * (F - (col.gather(0, i) - at)) / at.clamp_min(1e-20)
            xf = torch.where(hit.any(0, keepdim=True), xf, self.diag)
            xi = torch.maximum(xi, ((xf - self.axis[0]) / width + 0.5).clamp(0.0, 1.0))
            df = torch.minimum(df, self.axis[0] - xf)
        m = torch.zeros_like(xi)
        for ax, n in enumerate(self.shape):
            p = _edge_pad(xi, ax, 1)
            m += p.narrow(ax, 0, n) + p.narrow(ax, 2, n)
        self.xi, self.df = 0.5 * xi + 0.5 * (m / 6.0), df

    def fuv(self):
        nr, nu, nphi = _ray_budget(self.shape[2])[2]
        binr, kappa = self.diag / nr, float(self.P["kappa_fuv"])
        d = self._dirs(nu, nphi)
        g = torch.zeros_like(self.g0)
        for s in self.stars:
            o = [float(np.float32(v)) for v in s[:3]]
            n1 = int(self._range(o, d)[1].max())
            tau, att, ib = torch.zeros_like(d[0]), torch.zeros((nr, nu * nphi), device=self.dev, dtype=torch.float64), 0
            for n in range(n1):                                  # beyond a ray's own end the gas is empty
                r = (n + 0.5) * self.dx
                nv, x = self._sample([self.U[0], self.xi], [o[a] + d[a] * r for a in range(3)])
                tau = tau + kappa * nv * (1.0 - 0.92 * x) * self.dx
                nb = min(int(r / binr), nr)
                if nb > ib:
                    att[ib:nb] = torch.exp(-tau)
                    ib = nb
            att[ib:] = torch.exp(-tau)
            att = att.reshape(-1)
            for sl in range(0, self.shape[0], 64):
                r, u, phi = (v[sl:sl + 64] for v in self._polar(s))
                er, tr = self._lin(r / binr - 0.5, nr, False)
                eu, tu = self._lin((u + 1.0) * 0.5 * nu - 0.5, nu, False)
                ep, tp = self._lin(phi / (2.0 * math.pi) * nphi - 0.5, nphi, True)
                acc = torch.zeros_like(r)
                for a in range(2):
                    for b in range(2):
                        for c in range(2):
                            w = (tr if a else 1.0 - tr) * (tu if b else 1.0 - tu) * (tp if c else 1.0 - tp)
                            acc += w * att[(er[a] * nu + eu[b]) * nphi + ep[c]]
                g[sl:sl + 64] += s[3] * acc / (r * r).clamp_min(0.0004)
        if float(self.P.get("plane_flux", 0.0) or 0.0) > 0.0:
            dtau = kappa * self.U[0] * (1.0 - 0.92 * self.xi) * self.dx
            g += float(self.P.get("plane_fuv", 0.0) or 0.0) * torch.exp(-(torch.cumsum(dtau, 0) - 0.5 * dtau))
        self.g0 = g

    def voxels(self):
        def sstep(e0, e1, x):
            t = ((x - e0) / (e1 - e0)).clamp(0.0, 1.0)
            return t * t * (3.0 - 2.0 * t)
        rho, x = self.U[0], self.xi.clamp(0.0, 1.0)
        ha = (rho * x) ** 2
        df = self.df.to(torch.float16).double()                  # the fields the look reads are stored in 16 bits
        g = self.g0.to(torch.float16).double()
        if self.P.get("fp32_fields"):
            df, g = self.df, self.g0
        o3, s2 = ha * sstep(-0.03, -0.12, df), ha * sstep(-0.05, -0.005, df)
        dust = rho * (1.0 - x) + 0.08 * rho * x
        div = torch.zeros_like(rho)
        for ax, n in enumerate(self.shape):
            p = _edge_pad(self.U[1 + ax] / rho, ax, 1)
            div += (p.narrow(ax, 2, n) - p.narrow(ax, 0, n)) / (2.0 * self.dx)
        sh = (-div).clamp_min(0.0) * rho
        dg = dust * (g / (1.0 + g / LOOK["gs"]) + LOOK["ambient"])
        f = 1.0
        for X, L in zip(self.axis, self.L):
            f = f * sstep(0.0, LOOK["edge"], X / L) * sstep(0.0, LOOK["edge"], 1.0 - X / L)
        ch = [ha * LOOK["c_ha"][k] + o3 * LOOK["c_o3"][k] + s2 * LOOK["c_s2"][k] + dg * LOOK["c_dg"][k]
              + sh * LOOK["c_sh"][k] for k in range(3)] + [dust]
        v = torch.stack([(c * f).clamp_max(60000.0) for c in ch], dim=-1)
        for ax, n in enumerate(self.shape):
            p = _edge_pad(v, ax, 1)
            v = (p.narrow(ax, 0, n) + 4.0 * v + p.narrow(ax, 2, n)) / 6.0
        return v

    def state(self):
        return {"rho": self.U[0], "mx": self.U[1], "my": self.U[2], "mz": self.U[3], "xi": self.xi, "dfront": self.df}


def exact(case, seed):
    kind = case["kind"]
    if kind == "snapshot":
        return None                                              # bytes of a format: compared as they are
    out = []
    for ic in _scenes(case, seed, "cuda" if torch.cuda.is_available() else "cpu"):
        e = Exact(ic)
        every = max(int(e.P["ion_every"]), 3)                    # the fast budget's cadence
        if kind == "stir":
            A, B = (torch.as_tensor(f, device=e.dev, dtype=torch.float64) for f in ic["stir_fields"][:2])
            for _ in range(case["steps"]):
                e.pre_step(A, B, float(ic["stir_grid"][1]))
            out.append(e.state())
            continue
        if kind in ("ionize", "fuv", "render"):
            e.ionize()
        else:
            for _ in range(case["steps"]):
                e.step(every)
        if kind in ("fuv", "frame", "render"):
            e.fuv()
        if kind == "ionize":
            out.append({"xi": e.xi, "dfront": e.df})
        elif kind == "fuv":
            out.append({"g0": e.g0})
        elif kind == "frame":
            out.append({"voxels": e.voxels(), "g0": e.g0, "rho": e.U[0]})
        elif kind == "render":
            out.append({"voxels": e.voxels()})
        else:
            out.append(e.state())
    return out if kind == "batch" else out[0]
