"""The work that users of this library have it do, as measurable cases.

A case is one pass through the public entry points of the `wcsph` package:

kind "scene"     a simulation loop of one scene: `update` per frame (with
                 `set_box` before it when the box moves). io "device" starts
                 each pass from the same device-resident state (an episode
                 reset: a copy into the live fields on the context's stream)
                 and leaves the result on the device; io "host" restarts from
                 host arrays with `set_state` and reads the result back with
                 `get_state`, through pinned memory.
kind "ensemble"  many independent scenes advanced together (`BatchSimulator`),
                 as one persistent launch or as per-stage launches, and every
                 scene's state read back.
kind "rollout"   one iteration of an optimisation through the simulator:
                 `set_state`, `rollout_forward`, `rollout_backward`.
kind "keys"      `sort_keys_static` on device-resident Morton keys.

`exact` restates the path in 64 bits with plain torch (no code of this
repository): the neighbour sets and cells are those of the 32-bit inputs, all
sums are 64-bit.
"""
from __future__ import annotations

import ctypes
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "fluid-simulation_b200"))

import wcsph  # noqa: E402


def _scene(name, nx, ny, nz, radius, **kw):
    c = {"name": name, "kind": "scene", "nx": nx, "ny": ny, "nz": nz, "radius": radius,
         "spacing": 1.0,      # lattice spacing over 2r; 0.92 is the density of settled fluid
         "jitter": 0.1,       # over the radius
         "speed": 0.1,        # standard deviation of the velocities, m/s
         "walls": False,      # boundary particles on the box
         "sphere": 0.0,       # radius of a sampled sphere obstacle in the middle, m
         "tilt": 0.0,         # box rotation about z in degrees, set before each update
         "cfl": 0.0,          # CFL factor (0: fixed step)
         "reference": False,  # the reference application's constants (surface tension, small stiffness)
         "delta": 1e-3, "steps": 1, "io": "device"}
    c.update(kw)
    return c


def listed():
    return [
        # a small interactive scene or a unit test's: launches and latency count
        _scene("block_2k", 13, 13, 12, 0.01, walls=True, steps=4),
        # the reference's surface-tension application (30^3 particles, its constants, CFL
        # step), restarted from a saved state and read back
        _scene("droplet_27k", 30, 30, 30, 0.02, jitter=0.02, speed=0.3, cfl=0.4, reference=True, delta=0.01,
               steps=2, io="host"),
        # the 32^3 dam break in a walled tank of the tests and the benchmark
        _scene("dam_33k", 32, 32, 32, 0.01, walls=True, steps=4),
        # an odd-sized pool at rest density in a walled tank
        _scene("pool_79k", 43, 45, 41, 0.01, spacing=0.92, jitter=0.25, walls=True),
        # the benchmark's mesh-obstacle scene: walls and a sphere, CFL step
        _scene("obstacle_393k", 64, 96, 64, 0.005, walls=True, sphere=0.15, cfl=0.4, speed=0.5, io="host"),
        # the benchmark's headline scene: a million particles in a tilting box, no boundary particles
        _scene("tilting_1m", 128, 128, 64, 0.004, jitter=0.2, tilt=7.5, delta=5e-4),
        # a settled, disordered fluid with odd dimensions, as most steps of a long run meet it
        _scene("settled_700k", 97, 79, 91, 0.004, spacing=0.92, jitter=0.35, speed=0.2, delta=5e-4),
        # the largest: four million particles
        _scene("large_4m", 256, 128, 128, 0.0025, jitter=0.2, tilt=3.0, delta=2.5e-4),
        # ensembles of independent scenes (2,048 to 65,536 particles each): the default
        # persistent launch, and per-stage launches
        {"name": "ensemble_12", "kind": "ensemble", "first": 0, "scenes": 12, "persistent": True, "steps": 2},
        {"name": "ensemble_32_staged", "kind": "ensemble", "first": 12, "scenes": 32, "persistent": False, "steps": 2},
        # gradients of a rollout of the 32 x 32 x 16 block in a walled tank
        {"name": "rollout_16k", "kind": "rollout", "nx": 32, "ny": 32, "nz": 16, "radius": 0.01, "steps": 10,
         "every": 5},
        # the allocation-free sort at its capacity
        {"name": "keys_64k", "kind": "keys", "n": 65536, "bits": 24},
    ]


def draw(rng):
    u = rng.random()
    if u < 0.7:
        n = math.exp(rng.uniform(math.log(2000), math.log(3.5e6)))
        ax, ay = rng.uniform(0.6, 1.7), rng.uniform(0.6, 1.7)
        side = (n / (ax * ay)) ** (1 / 3)
        nx, ny, nz = (max(8, int(round(side * a))) for a in (ax, ay, 1.0))
        n = nx * ny * nz
        settled = rng.random() < 0.5
        small = n < 120000
        walls = rng.random() < (0.7 if small else 0.3)
        radius = 0.01 if n < 200000 else 0.005 if n < 800000 else 0.003
        c = {"kind": "scene", "nx": nx, "ny": ny, "nz": nz, "radius": radius,
             "spacing": round(rng.uniform(0.91, 0.95), 3) if settled else 1.0,
             "jitter": round(rng.uniform(0.1, 0.4), 3), "speed": round(rng.uniform(0.05, 0.5), 3),
             "walls": walls, "sphere": 0.0, "tilt": round(rng.uniform(1, 15), 2) if rng.random() < 0.3 else 0.0,
             "cfl": 0.0, "reference": False, "delta": 1e-3 if radius == 0.01 else 5e-4 if radius == 0.005 else 2.5e-4,
             "steps": rng.choice([1, 2, 4]) if small else 1, "io": "device"}
        if rng.random() < 0.25:
            c.update(cfl=0.4, io="host")
        return c
    if u < 0.85:
        return {"kind": "ensemble", "first": rng.randrange(200), "scenes": rng.randrange(5, 33),
                "persistent": rng.random() < 0.5, "steps": rng.choice([1, 2])}
    if u < 0.95:
        return {"kind": "rollout", "nx": rng.randrange(16, 37), "ny": rng.randrange(16, 37),
                "nz": rng.randrange(12, 25), "radius": 0.01, "steps": rng.randrange(6, 13), "every": rng.randrange(3, 7)}
    return {"kind": "keys", "n": int(math.exp(rng.uniform(math.log(500), math.log(65536)))),
            "bits": rng.choice([15, 18, 21, 24, 27, 30])}


# ---------------------------------------------------------------- inputs --
def _params(c):
    r = c["radius"]
    if c.get("reference"):
        # the reference's own constants; its application pushes the fluid up
        p = wcsph.default_params(particle_radius=r, external_force=wcsph.FORCE_CONSTANT,
                                 external_force_param=(0.0, 9.81, 0.0))
        p.cfl_factor = c["cfl"]
        return p
    # textbook Tait stiffness 1000 in the reference's normalisation of the spiky gradient
    k = 1000.0 * (4.0 * r) ** 6
    return wcsph.default_params(particle_radius=r, stiffness=k, viscosity=0.01, cfl_factor=c.get("cfl", 0.0),
                                max_time_step=c.get("delta", 1e-3), min_time_step=1e-5,
                                surface_tension=0.0 if c["kind"] == "rollout" else 0.13)


def _lattice(c, rng, spacing, jitter):
    """The fluid block with its corner at the box corner, float32 [n, 4]."""
    r = c["radius"]
    s = 2 * r * spacing
    g = np.stack(np.meshgrid(*(np.arange(c[k], dtype=np.float32) for k in ("nx", "ny", "nz")), indexing="ij"), -1)
    x = np.empty((g.size // 3, 4), np.float32)
    x[:, :3] = g.reshape(-1, 3) * np.float32(s)
    x[:, :3] += np.float32(r * (1 + jitter))
    x[:, :3] += rng.uniform(-jitter * r, jitter * r, (len(x), 3)).astype(np.float32)
    x[:, 3] = 1
    return x


def _inputs(c, seed):
    """Positions, velocities, box corners and boundary particles of a single scene."""
    rng = np.random.default_rng(seed)
    r = c["radius"]
    roll = c["kind"] == "rollout"
    pos = _lattice(c, rng, c.get("spacing", 1.0), c.get("jitter", 0.1))
    vel = np.zeros_like(pos)
    vel[:, :3] = rng.standard_normal((len(pos), 3), dtype=np.float32) * np.float32(c.get("speed", 0.1))
    ext = np.array([c[k] * 2 * r * c.get("spacing", 1.0) + 2 * r for k in ("nx", "ny", "nz")])
    ext *= np.array([1.6, 1.3, 1.6 if roll else 1.0])   # room to spread
    mn = np.zeros(3)
    if not c.get("walls", roll):   # around the origin
        pos[:, :3] -= (ext / 2).astype(np.float32)
        mn = -ext / 2
    mx = mn + ext
    bnd = None
    if c.get("walls", roll):
        bnd = wcsph.sample_box_walls(mn, mx, 2 * r)
        if c.get("sphere"):
            mid = np.array([ext[0] / 2, ext[1] / 2, ext[2] / 2])
            bnd = np.concatenate([bnd, wcsph.sample_icosphere(mid, c["sphere"], 4, 2 * r)])
    return pos, vel, mn, mx, bnd


def _model(c):
    return wcsph.rotation_z(math.radians(c["tilt"])) if c.get("tilt") else None


def _ensemble(c, seed):
    """Scenes first .. first + scenes - 1 of the benchmark's ensemble (their sizes, boxes, gravity and
    viscosity), with positions and velocities disturbed by the seed."""
    rng = np.random.default_rng(seed)
    pres = [wcsph.preset_ensemble(1, c["first"] + k) for k in range(c["scenes"])]
    for p in pres:
        p.pos[:, :3] += rng.uniform(-0.001, 0.001, (len(p.pos), 3)).astype(np.float32)
        p.vel[:, :3] = rng.standard_normal((len(p.pos), 3), dtype=np.float32) * np.float32(0.1)
    return pres


def _morton_keys(c, seed):
    """Morton keys as the step computes them, of cells spread over a box of 2^(bits / 3) cells per axis."""
    rng = np.random.default_rng(seed)
    per = 1 << (c["bits"] // 3)
    cells = rng.integers(-per // 2, per // 2, (c["n"], 3)) + (1 << 20)
    return _interleave(torch.from_numpy(cells))


def _interleave(cells):
    key = torch.zeros(len(cells), dtype=torch.int64, device=cells.device)
    for b in range(21):
        for d in range(3):
            key |= ((cells[:, d] >> b) & 1) << (3 * b + d)
    return key


class _DeviceArray:
    """A borrowed device pointer; keeps its owner alive as long as a tensor views it."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3}


class _Scene:
    """A simulator and what a program keeps beside it."""

    def __init__(self, c, seed):
        pos, vel, mn, mx, bnd = _inputs(c, seed)
        self.c = c
        self.box = wcsph.box(mn, mx, _model(c))
        self.sim = wcsph.CUDASPHSimulator(_params(c), pos, wcsph.box(mn, mx), fluid_vel=vel, boundary_pos=bnd)
        self.n = len(pos)
        if c.get("io") == "device":
            self.stream = torch.cuda.ExternalStream(self.sim.stream_handle())
            self.pos0, self.vel0 = torch.from_numpy(pos).cuda(), torch.from_numpy(vel).cuda()
            torch.cuda.current_stream().synchronize()
            self.views = {}
        else:
            pin = lambda a: torch.from_numpy(a).pin_memory().numpy()  # noqa: E731
            self.pos0, self.vel0 = pin(pos), pin(vel)
            self.out = pin(np.zeros_like(pos)), pin(np.zeros_like(vel))

    def field(self, name):
        """The live field on the device as a tensor (the pointer is asked for anew at each use)."""
        p = ctypes.c_void_p()
        sim = self.sim
        sim._c(sim._lib.wcsph_get_device_field(sim._ctx, wcsph.FIELD[name], ctypes.byref(p)))
        t = self.views.get(name)
        if t is None or t.data_ptr() != p.value:
            shape = (self.n,) if name == "density" else (self.n, 4)
            t = self.views[name] = torch.as_tensor(_DeviceArray(sim, p.value, shape, "<f4"), device="cuda")
        return t


def prepare(case, seed):
    kind = case["kind"]
    if kind == "scene":
        return _Scene(case, seed)
    if kind == "ensemble":
        pres = _ensemble(case, seed)
        specs = [wcsph.BatchSceneSpec(fluid_pos=p.pos, fluid_vel=p.vel, box=p.box, gravity=tuple(p.params.gravity),
                                      viscosity=p.params.viscosity, boundary_pos=p.bpos) for p in pres]
        sim = wcsph.BatchSimulator(pres[0].params, specs)
        sim.set_persistent(case["persistent"])
        return {"kind": kind, "case": case, "sim": sim}
    if kind == "rollout":
        s = _Scene(case, seed)
        target = s.pos0.copy()
        target[:, 0] += 0.2
        target[:, 2] += 0.1
        return {"kind": kind, "case": case, "scene": s, "target": target}
    keys = _morton_keys(case, seed).cuda()
    return {"kind": kind, "keys": keys, "perm": torch.empty(len(keys), dtype=torch.int32, device="cuda")}


# ------------------------------------------------------------------ pass --
def run(state):
    if isinstance(state, _Scene):
        c, sim = state.c, state.sim
        device = c["io"] == "device"
        if device:
            with torch.cuda.stream(state.stream):
                state.field("position").copy_(state.pos0, non_blocking=True)
                state.field("velocity").copy_(state.vel0, non_blocking=True)
        else:
            sim.set_state(state.pos0, state.vel0)
        for _ in range(c["steps"]):
            if c["tilt"]:
                sim.set_box(state.box)
            sim.update(c["delta"])
        if device:
            return {k: state.field(k) for k in ("position", "velocity", "density")}
        pos, vel = sim.get_state(out=state.out)
        return {"position": pos, "velocity": vel}
    if state["kind"] == "ensemble":
        sim = state["sim"]
        sim.step_n(state["case"]["steps"], 1e-3)
        got = [sim.get_state(k) for k in range(state["case"]["scenes"])]
        return {"position": np.concatenate([g[0] for g in got]), "velocity": np.concatenate([g[1] for g in got])}
    if state["kind"] == "rollout":
        c, s = state["case"], state["scene"]
        s.sim.set_state(s.pos0, s.vel0)
        loss = s.sim.rollout_forward(c["steps"], 1e-3, c["every"], state["target"])
        gv, gnu, gk = s.sim.rollout_backward()
        return {"loss": loss, "grad_velocity": gv, "grad_viscosity": gnu, "grad_stiffness": gk}
    keys, perm = state["keys"], state["perm"]
    wcsph.sort_keys_static(keys.data_ptr(), len(keys), perm.data_ptr(), torch.cuda.current_stream().cuda_stream)
    return perm


def _particles(case):
    if case["kind"] == "ensemble":
        return case["scenes"] * 18000   # the mean of the log-uniform counts
    return case["nx"] * case["ny"] * case["nz"]


def work(case):
    if case["kind"] == "keys":
        return {"bytes": 12 * case["n"], "flops": 0}
    n = _particles(case)
    # state in and out and the density; about 33 neighbours a particle, 135 operations a pair and step
    flops = 135 * 33 * n * case["steps"]
    if case["kind"] == "rollout":
        return {"bytes": 16 * 4 * n, "flops": 4 * flops}
    return {"bytes": (64 + (4 if case.get("io") == "device" else 0)) * n, "flops": flops}


# ----------------------------------------------------------------- 64 bits --
def _f32(x):
    return np.float32(x)


class _Constants:
    """The derived constants of a step; cells and the neighbour predicate use the 32-bit h."""

    def __init__(self, p, gravity=None, viscosity=None):
        s = _f32(2) * _f32(p.particle_radius)
        self.h32 = _f32(2) * s
        self.h2_32 = float(self.h32 * self.h32)
        self.cs32 = float(self.h32 * _f32(p.cell_size_mult))
        self.r, self.s, self.h = float(p.particle_radius), float(s), float(self.h32)
        self.rho0, self.k, self.gamma = float(p.rest_density), float(p.stiffness), float(p.exponent)
        self.most = float(p.max_density_ratio)
        self.m = self.rho0 * self.s ** 3 * 0.8
        self.nu = float(p.viscosity) if viscosity is None else float(viscosity)
        self.alpha = float(p.surface_tension)
        self.g = [float(v) for v in (p.gravity if gravity is None else gravity)]
        if p.external_force == wcsph.FORCE_CONSTANT:
            self.g = [a + float(b) for a, b in zip(self.g, p.external_force_param)]
        h3 = math.pi * self.h ** 3
        self.cw, self.cg, self.coh = 8 / h3, 48 / h3, 32 / h3
        self.sp = -45 / (math.pi * self.h ** 9)
        self.buf, self.elastic = self.r * float(p.collision_buffer_mult), float(p.elasticity)
        self.cfl, self.max_dt, self.min_dt = float(p.cfl_factor), float(p.max_time_step), float(p.min_time_step)
        self.np_max = float(p.non_pressure_max_time_step)


def _cells(x, cs):
    """Cells of 32-bit positions, offset to be positive."""
    q = x[:, :3].float() / torch.tensor(cs, dtype=torch.float32, device=x.device)
    return torch.floor(q).long() + (1 << 20)


def _flat(cell):
    return cell[:, 0] | cell[:, 1] << 21 | cell[:, 2] << 42


def _pairs(xi, xj, cs, h2, same):
    """(i, j) of all pairs within h by the 32-bit predicate fma(z, z, fma(x, x, y y)) <= h^2."""
    ci = _cells(xi, cs)
    fj, order = torch.sort(_flat(_cells(xj, cs)), stable=True)
    xj32, xi32 = xj[order].float(), xi.float()
    ii, jj = [], []
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dz in (-1, 0, 1):
                f = _flat(ci + torch.tensor([dx, dy, dz], device=xi.device))
                lo, hi = torch.searchsorted(fj, f), torch.searchsorted(fj, f, right=True)
                most = int((hi - lo).max())
                for t in range(most):
                    i = torch.nonzero(lo + t < hi).flatten()
                    j = lo[i] + t
                    d = xi32[i, :3] - xj32[j, :3]
                    y2 = (d[:, 1] * d[:, 1]).double()
                    d = d.double()
                    r2 = (d[:, 2] ** 2 + (d[:, 0] ** 2 + y2).float().double()).float()
                    ok = r2.double() <= h2
                    if same:
                        ok &= order[j] != i
                    ii.append(i[ok])
                    jj.append(order[j[ok]])
    return torch.cat(ii), torch.cat(jj)


def _sum(n, i, v):
    out = torch.zeros((n,) + v.shape[1:], dtype=v.dtype, device=v.device)
    return out.index_add(0, i, v)


def _length(d):
    r2 = (d * d).sum(1)
    return torch.sqrt(torch.clamp(r2, min=1e-30)), r2


def _w(q):
    return torch.where(q <= 0.5, 6 * q ** 3 - 6 * q ** 2 + 1, torch.where(q <= 1, 2 * (1 - q) ** 3, torch.zeros_like(q)))


def _boundary_masses(b, K):
    i, j = _pairs(b, b, K.h, K.h2_32, True)
    rl, _ = _length(b[i, :3].double() - b[j, :3].double())
    return K.rho0 / (K.cw + _sum(len(b), i, K.cw * _w(rl / K.h)))


def _step(x, v, K, box, delta, bnd, nu=None, stiff=None):
    """One step in 64 bits: (x, v, rho, order), sorted by cell; differentiable in x, v, nu and stiff."""
    nu = K.nu if nu is None else nu
    stiff = K.k if stiff is None else stiff
    vmax = float(v.detach()[:, :3].square().sum(1).max().sqrt())
    dt = min(max(delta, K.min_dt), K.max_dt)
    if K.cfl > 0:
        dt = K.max_dt if vmax < 1e-9 else min(dt, K.cfl * K.s / vmax)
    np_dt = min(delta, K.np_max)
    order = torch.sort(_interleave(_cells(x.detach(), K.cs32)), stable=True)[1]
    x, v = x[order], v[order]
    n = len(x)
    at, vel = x[:, :3], v[:, :3]
    i, j = _pairs(x.detach(), x.detach(), K.cs32, K.h2_32, True)
    d = at[i] - at[j]
    rl, r2 = _length(d)
    q = rl / K.h
    inside = (q >= 1e-9) & (q <= 1)
    zero = torch.zeros_like(q)
    rho = K.m * (K.cw + _sum(n, i, K.cw * _w(q)))
    if bnd is not None:
        xb, mb = bnd
        bi, bj = _pairs(x.detach(), xb, K.h, K.h2_32, False)
        bd = at[bi] - xb[bj, :3].double()
        bl, _ = _length(bd)
        bq = bl / K.h
        rho = rho + _sum(n, bi, mb[bj] * K.cw * _w(bq))
    p = stiff * (torch.clamp(rho / K.rho0, 1.0, K.most) ** K.gamma - 1)
    sg = torch.where(inside, K.sp * (1 - q) ** 2 / (K.h * rl), zero)
    cg = torch.where(inside, torch.where(q <= 0.5, K.cg * q * (3 * q - 2), -K.cg * (1 - q) ** 2) / (K.h * rl), zero)
    pr = p / rho ** 2
    ap = K.m * _sum(n, i, -((pr[i] + pr[j]) * sg)[:, None] * d)
    if bnd is not None:
        bs = torch.where((bq >= 1e-9) & (bq <= 1), K.sp * (1 - bq) ** 2 / (K.h * bl), torch.zeros_like(bq))
        ap = ap - _sum(n, bi, (mb[bj] * (pr[bi] + p[bi] / K.rho0 ** 2) * bs)[:, None] * bd)
    vr = ((vel[i] - vel[j]) * d).sum(1)
    lap = _sum(n, i, (vr * cg / (rho[j] * (r2 + 0.01 * K.h * K.h)))[:, None] * d)
    anp = torch.tensor(K.g, dtype=torch.float64, device=x.device) + nu * 10 * K.m * lap
    if K.alpha:
        normal = K.h * K.m * _sum(n, i, (cg / rho[j])[:, None] * d)
        a = (q * (1 - q)) ** 3
        c = K.coh * torch.where(q <= 0.5, 2 * a - 1 / 64, torch.where(q <= 1, a, zero))
        f = ((K.m * c / rl)[:, None] * d + normal[i] - normal[j]) / (rho[i] + rho[j])[:, None]
        anp = anp - K.alpha * 2 * K.rho0 * _sum(n, i, torch.where((r2 > 1e-6)[:, None], f, torch.zeros_like(f)))
    vel = vel + np_dt * anp + dt * ap
    at = at + dt * vel
    mn, mx, M, Mi = box
    loc, u = at @ Mi[:3, :3].T + Mi[:3, 3], vel @ Mi[:3, :3].T
    low, high = loc.detach() - K.buf < mn, loc.detach() + K.buf > mx
    hit = (low | high).any(1, keepdim=True)
    loc = torch.where(low, mn + K.r, torch.where(high, mx - K.r, loc))
    u = torch.where(low | high, -K.elastic * u, u)
    at = torch.where(hit, loc @ M[:3, :3].T + M[:3, 3], at)
    vel = torch.where(hit, u @ M[:3, :3].T, vel)
    return torch.cat([at, x[:, 3:]], 1), torch.cat([vel, v[:, 3:]], 1), rho, order


def _box64(box, dev):
    t = lambda v: torch.tensor([float(a) for a in v], dtype=torch.float64, device=dev)  # noqa: E731
    return t(box.min), t(box.max), t(box.model).reshape(4, 4).T, t(box.model_inv).reshape(4, 4).T


def exact(case, seed):
    kind = case["kind"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    up = lambda a: torch.from_numpy(a).to(dev)  # noqa: E731
    if kind == "keys":
        return None
    if kind == "ensemble":
        out = []
        for p in _ensemble(case, seed):
            K = _Constants(p.params, p.params.gravity, p.params.viscosity)
            x, v, b = up(p.pos).double(), up(p.vel).double(), up(p.bpos)
            bnd = (b, _boundary_masses(b, K))
            for _ in range(case["steps"]):
                x, v, _, _ = _step(x, v, K, _box64(p.box, dev), 1e-3, bnd)
            out.append((x, v))
        return {"position": torch.cat([o[0] for o in out]), "velocity": torch.cat([o[1] for o in out])}
    pos, vel, mn, mx, b = _inputs(case, seed)
    K = _Constants(_params(case))
    bnd = None if b is None else (up(b), _boundary_masses(up(b), K))
    x, v = up(pos).double(), up(vel).double()
    if kind == "scene":
        box = _box64(wcsph.box(mn, mx, _model(case)), dev)
        for _ in range(case["steps"]):
            x, v, rho, _ = _step(x, v, K, box, float(_f32(case["delta"])), bnd)
        out = {"position": x, "velocity": v}
        return out | {"density": rho} if case["io"] == "device" else out
    box = _box64(wcsph.box(mn, mx), dev)
    K.cfl = 0.0
    K.max_dt = K.min_dt = float(_f32(1e-3))   # the rollout's step is fixed
    v = v.requires_grad_()
    nu = torch.tensor(K.nu, dtype=torch.float64, device=dev, requires_grad=True)
    stiff = torch.tensor(K.k, dtype=torch.float64, device=dev, requires_grad=True)
    ids = torch.arange(len(x), device=dev)
    target = x[:, :3] + torch.tensor([0.2, 0.0, 0.1], dtype=torch.float64, device=dev)
    y, w = x, v
    for _ in range(case["steps"]):
        y, w, _, order = _step(y, w, K, box, K.max_dt, bnd, nu, stiff)
        ids = ids[order]
    loss = (y[:, :3] - target[ids]).square().sum() / len(x)
    gv, gnu, gk = torch.autograd.grad(loss, (v, nu, stiff))
    return {"loss": loss.detach(), "grad_velocity": gv, "grad_viscosity": gnu, "grad_stiffness": gk}
