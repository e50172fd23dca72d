"""What a user of this framework has it do, as measurable cases.

Each case is a dict of plain values; ``prepare`` builds the solver objects a driver has in hand,
``run`` is one pass of the driver's loop through the public classes, ``exact`` the same pass in plain
torch / numpy at 64 bits.  Sizes follow ``lbdem_taichi_b200.cases`` (single settling sphere, dense
suspension, large channel, packed bed), the tests' small ragged lattices and the drag-gradient
channel of the benchmark; ``draw`` spreads them over the same ranges.

Kinds:
  couple  particles in a periodic box or a channel: collide, stream, DEM sub-steps, through ``run()``
          or as the plain driver loop with one ``run_simulation()`` per sub-step
  shear   suspension between moving walls, stress diagnostics after every stream
  bed     frozen packed bed, Ladd velocity inlet and Zou-He pressure outlet
  grad    drag gradient on a frozen bed (reverse mode)
  dem     the DEM solver alone on a dense bed in contact
  fluid   the lattice classes alone (BasicLattice3D, ForcedLattice3D)

Populations come back as the device holds them (scaled deviations in x-blocks of 32, include/lbdem.h).
Quantities that FP32 kernels compute -- hydrodynamic force and torque, the velocities they drive,
stresses, gradients -- come back in FP32, also where they are summed or kept in FP64 fields; the
positions, and everything of the DEM alone, in FP64.
"""
from __future__ import annotations

import math

import numpy as np
import torch

W = [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12
CQ = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, -1, 0),
      (1, -1, 0), (-1, 1, 0), (1, 0, 1), (-1, 0, -1), (1, 0, -1), (-1, 0, 1), (0, 1, 1), (0, -1, -1), (0, 1, -1),
      (0, -1, 1)]
OPP = [0] + [q + 1 if q % 2 else q - 1 for q in range(1, 19)]
FLUID, OBSTACLE, MOVING = 1, 8, 32
INLET_LEFT, OUTLET_RIGHT = 262144 | 8192, 256 | 4096
SCALE = {"f32": 1.0, "f16": 4096.0, "bf16": 1.0}
FLUID_FORCE = 1e-6
WALL_U = 5e-3
INLET_U = 2e-3
YOUNG, POISSON, FRICTION, RESTITUTION = 1e5, 0.3, 0.3, 0.9
LIN_KN, LIN_KS, LIN_DN, LIN_MU = 4.5e3, 2.5e3, 0.3, 0.15


def _couple(**kw):
    c = dict(kind="couple", nx=64, ny=64, nz=128, n=1, dmin=12.0, dmax=12.0, walls=True, storage="f32", lag16=False,
             smag="reference", cs=0.1, tau=0.6, force=False, wrapped=False, loop="run", steps=8, sub=10)
    c.update(kw)
    return c


def listed():
    return [
        # the settling driver's own loop, unchanged but for its imports: one lattice step and ten run_simulation()
        # calls; latency and launches are all there is
        dict(_couple(loop="driver", steps=1), name="settle_driver"),
        # the same set-up through run(): a long settling run, where the sphere's DEM chain is most of a step
        dict(_couple(steps=10), name="settle_run"),
        # dense suspension, the benchmark's configuration, FP32
        dict(_couple(nx=256, ny=256, nz=256, n=2000, dmin=8.0, dmax=12.0, walls=False, force=True, steps=4),
             name="suspension_f32"),
        # the same in FP16 population storage, the form that the metric is quoted for
        dict(_couple(nx=256, ny=256, nz=256, n=2000, dmin=8.0, dmax=12.0, walls=False, force=True, steps=4,
                     storage="f16"), name="suspension_f16"),
        # half of the large LES channel: many small spheres, z walls (per-cell link masks), low viscosity; the largest
        dict(_couple(nx=512, ny=256, nz=256, n=10000, dmin=6.0, dmax=10.0, force=True, tau=0.51, cs=0.12, steps=2),
             name="channel_f32"),
        # ragged lattice, BF16 storage, spheres mapped and in contact across the periodic faces
        dict(_couple(nx=203, ny=97, nz=118, n=260, dmin=7.0, dmax=9.0, walls=False, force=True, wrapped=True, tau=0.56,
                     storage="bf16", steps=6), name="ragged_bf16_wrapped"),
        # shear rheology: moving walls, compute_stress() after every stream, a plane average at the end
        dict(kind="shear", name="shear_stress", nx=128, ny=96, nz=130, n=150, dmin=10.0, dmax=12.0, storage="f32",
             cs=0.1, tau=0.7, steps=6, sub=10),
        # packed-bed pressure drop at half the driver's resolution, started in uniform flow: open boundaries, frozen bed
        dict(kind="bed", name="bed_open_f32", nx=362, ny=122, nz=122, n=1400, d=12.0, storage="f32", tau=0.68, steps=6),
        # one drag gradient on the 500-sphere bed of the gradient benchmark, shortened
        dict(kind="grad", name="gradient", nx=128, ny=128, nz=128, n=500, d=10.0, tau=0.6, steps=60, every=20),
        # the DEM alone: a dense bed under gravity, every sphere in contact with its neighbours
        dict(kind="dem", name="dem_bed", n=8000, d=10.0, model="hertz", sub=10, jitter=2e-5),
        # plain fluid channel on an odd size, BGK with a body force
        dict(kind="fluid", name="forced_channel", nx=250, ny=131, nz=96, cls="forced", storage="f32", tau=0.8, walls=True,
             steps=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["couple"] * 5 + ["shear", "bed", "grad", "dem", "fluid"])
    if kind == "dem":
        return dict(kind=kind, n=_log(rng, 30, 8000), d=round(rng.uniform(6.0, 14.0), 3), model=rng.choice(["hertz", "linear"]),
                    sub=rng.choice([1, 7, 10, 25]), jitter=2e-5)
    # lattices of 30 thousand to 15 million cells, any aspect, odd sizes
    cells = _log(rng, 3e4, {"grad": 1.5e6, "shear": 3e6, "bed": 4e6}.get(kind, 1.5e7))
    a, b = rng.uniform(0.6, 1.7), rng.uniform(0.6, 1.7)
    e = cells ** (1 / 3)
    nx, ny = max(24, min(700, int(e * a))), max(24, min(500, int(e * b)))
    nz = max(26, min(500, int(cells / (nx * ny))))
    c = dict(kind=kind, nx=nx, ny=ny, nz=nz)
    if kind == "fluid":
        return dict(c, cls=rng.choice(["forced", "basic"]), storage=rng.choice(["f32", "f16", "bf16"]),
                    tau=round(rng.uniform(0.52, 1.2), 3), walls=rng.random() < 0.6, steps=rng.choice([4, 6, 8]))
    d = round(rng.uniform(5.0, 12.0), 2)
    if kind in ("bed", "grad"):
        room = _room((nx - 48 if kind == "bed" else nx, ny, nz), d + 0.6)
        c = dict(c, n=max(1, int(room * rng.uniform(0.2, 0.9))), d=d, tau=round(rng.uniform(0.55, 1.0), 3))
        if kind == "bed":
            return dict(c, nx=max(nx, 96), storage=rng.choice(["f32", "f16"]), steps=rng.choice([2, 4, 6]))
        return dict(c, steps=rng.choice([8, 15, 24]), every=rng.choice([4, 10]))
    dmax = round(d * rng.uniform(1.0, 1.4), 2)
    n = max(1, int(np.prod(_slots((nx, ny, nz), dmax, 1.0, nz - 1.0)) * rng.uniform(0.1, 0.9)))
    c = dict(c, n=n, dmin=d, dmax=dmax, tau=round(rng.uniform(0.51, 0.9), 3), cs=0.1, storage=rng.choice(["f32", "f16", "bf16"]))
    if kind == "shear":
        return dict(c, steps=rng.choice([2, 4, 6]), sub=rng.choice([1, 5, 10]))
    smag = rng.choice(["reference", "reference", "local", "off"])
    lag16 = c["storage"] == "f32" and smag == "reference" and rng.random() < 0.3
    wrapped = min(nx, ny) >= 8 * dmax + 2 and rng.random() < 0.25
    loop = rng.choice(["run", "run", "driver"])
    return _couple(**dict(c, lag16=lag16, smag=smag, walls=wrapped or rng.random() < 0.6, force=rng.random() < 0.6,
                          wrapped=wrapped, loop=loop, steps=rng.choice([2, 4, 6]), sub=rng.choice([1, 4, 10])))


# ------------------------------------------------------------------------------------------ inputs
def _room(shape, s):
    return max(0, int(shape[0] // s)) * max(0, int(shape[1] // s)) * max(0, int(shape[2] // s))


def _slots(shape, dmax, zlo, zhi):
    """Boxes of 2 x 1 x 1 sphere boxes along x, y and z."""
    s = dmax + 0.6
    return np.array([int((shape[0] - 1.0) // (2 * s)), int((shape[1] - 1.0) // s), int((zhi - zlo - 1.0) // s)])


def _spheres(rng, shape, n, dmin, dmax, zlo, zhi, pairs=0.2):
    """n spheres without overlap but for a share that touch in pairs (a suspension in motion has contacts of a few
    1e-4 lattice units' depth): random slots of 2 x 1 x 1 sphere boxes, a random place in each."""
    s = dmax + 0.6
    lo = np.array([0.5, 0.5, zlo + 0.5])
    m = _slots(shape, dmax, zlo, zhi)
    slots = int(np.prod(m))
    p = max(int(pairs * n / 2), n - slots)
    if 2 * p > n or n - p > slots:
        raise ValueError("too many spheres for the box")
    at = rng.permutation(slots)[:n - p]
    base = lo + np.stack([at % m[0], (at // m[0]) % m[1], at // (m[0] * m[1])], 1) * np.array([2 * s, s, s])
    r = 0.5 * rng.uniform(dmin, dmax, n)
    pos = np.empty((n, 3))
    ra, rb = r[:p], r[p:2 * p]
    pos[:p] = base[:p] + np.stack([ra, np.full(p, 0.5 * s), np.full(p, 0.5 * s)], 1) + rng.uniform(0.0, 0.02, (p, 3))
    tilt = np.concatenate([np.ones((p, 1)), rng.uniform(-0.03, 0.03, (p, 2))], 1)
    tilt /= np.linalg.norm(tilt, axis=1, keepdims=True)
    pos[p:2 * p] = pos[:p] + tilt * (ra + rb - rng.uniform(0.0, 5e-4, p))[:, None]
    k = n - 2 * p
    rs = r[2 * p:, None]
    pos[2 * p:] = base[p:] + rs + rng.uniform(0.0, 1.0, (k, 3)) * (np.array([2 * s, s, s]) - 2 * rs)
    o = rng.permutation(n)
    return pos[o], r[o]


def _inputs(c, seed):
    """Particle arrays of a case: centres, radii, velocities, angular velocities, masses (numpy, from the seed)."""
    rng = np.random.default_rng(seed)
    nx, ny, nz = c.get("nx"), c.get("ny"), c.get("nz")
    n = c["n"]
    rho = 2.0
    if c["kind"] == "dem":
        side = max(1, math.ceil((n / 2.0) ** (1 / 3)))
        s = c["d"] * (1 - 1e-4)
        i = np.arange(n)
        pos = np.stack([(i % side + 0.5), ((i // side) % side + 0.5), (i // side ** 2) + 0.5], 1) * s
        pos += rng.uniform(-1.0, 1.0, (n, 3)) * c["jitter"] * c["d"]
        r = np.full(n, 0.5 * c["d"])
    elif c["kind"] in ("bed", "grad"):
        s = c["d"] + 0.6
        x0 = 24.0 if c["kind"] == "bed" else 0.3
        zlo = 0.3 if c["kind"] == "bed" else 1.3
        m = np.array([int((nx - 2 * x0) // s), int(ny // s), int((nz - 2 * zlo) // s)])
        at = rng.permutation(int(np.prod(m)))[:n]
        n = len(at)
        pos = np.stack([at % m[0], (at // m[0]) % m[1], at // (m[0] * m[1])], 1) * s + 0.5 * s
        pos += rng.uniform(-0.25, 0.25, (n, 3)) + np.array([x0, 0.0, zlo])
        r = np.full(n, 0.5 * c["d"])
    elif n == 1:
        pos = np.array([[nx / 2 + rng.uniform(-0.5, 0.5), ny / 2 + rng.uniform(-0.5, 0.5),
                         max(nz - 6.0 - c["dmax"], nz / 2)]])
        r = np.array([0.5 * rng.uniform(c["dmin"], c["dmax"])])
        rho = 2.5
    else:
        walls = c["kind"] == "shear" or c["walls"]
        pos, r = _spheres(rng, (nx, ny, nz), n, c["dmin"], c["dmax"], 1.0 if walls else 0.0, nz - 1.0 if walls else float(nz))
        if c.get("wrapped"):    # spheres across the periodic faces
            pos[:, 0] = np.mod(pos[:, 0] + rng.uniform(0.0, nx), nx)
            pos[:, 1] = np.mod(pos[:, 1] + rng.uniform(0.0, ny), ny)
    still = c["kind"] in ("bed", "grad")
    vel = np.zeros((n, 3)) if still else rng.normal(0.0, 1e-3, (n, 3))
    omega = np.zeros((n, 3)) if still else rng.normal(0.0, 1e-3, (n, 3))
    return pos, r, vel, omega, rho * 4.0 / 3.0 * np.pi * r ** 3


def _domain(c, r):
    if c["kind"] != "dem":
        return (0.0, float(c["nx"]), 0.0, float(c["ny"]), 0.0, float(c["nz"]))
    side = max(1, math.ceil((c["n"] / 2.0) ** (1 / 3)))
    s, high = c["d"] * (1 - 1e-4), -(-c["n"] // side ** 2)
    return (-2.0 * c["d"], (side + 2.0) * s, -2.0 * c["d"], (side + 2.0) * s, 0.0, (high + 4.0) * s)


def _gravity(c):
    if c["kind"] == "dem":
        return (0.0, 0.0, -1e-4)
    if c["kind"] in ("bed", "grad", "shear"):
        return (0.0, 0.0, 0.0)
    return (0.0, 0.0, -1e-5 * 0.6) if c["n"] == 1 else (FLUID_FORCE, 0.0, 0.0)


def _periodic(c):
    if c["kind"] in ("dem", "bed"):
        return (False, c["kind"] == "bed", c["kind"] == "bed")
    return (True, True, not (c["kind"] in ("shear", "grad") or c["walls"]))


def _cell_types(c):
    ct = np.full((c["nx"], c["ny"], c["nz"]), FLUID, np.int32)
    if c["kind"] == "bed":
        ct[0] = INLET_LEFT
        ct[-1] = OUTLET_RIGHT
    elif c["kind"] == "shear":
        ct[:, :, 0] = ct[:, :, -1] = MOVING
    elif c["kind"] == "grad" or c.get("walls"):
        ct[:, :, 0] = ct[:, :, -1] = OBSTACLE
    else:
        return None
    return ct


def _start_velocity(c, seed):
    """Initial fluid velocity of the fluid-only cases (x, y, z, 3): a smooth random flow."""
    rng = np.random.default_rng(seed)
    x, y, z = (np.arange(m) * (2 * np.pi / m) for m in (c["nx"], c["ny"], c["nz"]))
    v = np.zeros((c["nx"], c["ny"], c["nz"], 3))
    for a in range(3):
        k, p = rng.integers(1, 4, 3), rng.uniform(0, 2 * np.pi, 3)
        v[..., a] = 0.02 * (np.sin(k[0] * x + p[0])[:, None, None] * np.cos(k[1] * y + p[1])[None, :, None]
                            * np.cos(k[2] * z + p[2])[None, None, :])
    return v.astype(np.float32)


def _build_dem(c, seed):
    from lbdem_taichi_b200.cases import make_dem
    from lbdem_taichi_b200.dem3d.demconfig import HertzContactConfig, LinearContactConfig
    pos, r, vel, omega, mass = _inputs(c, seed)
    linear = c["kind"] == "bed" or c.get("model") == "linear"
    contact = (LinearContactConfig(stiffness_normal=LIN_KN, stiffness_tangential=LIN_KS, damping_normal=LIN_DN,
                                   damping_tangential=0.2, pp_friction=LIN_MU, pw_friction=LIN_MU) if linear else
               HertzContactConfig(pp_friction=FRICTION, pw_friction=FRICTION, pp_restitution=RESTITUTION,
                                  pw_restitution=RESTITUTION))
    sub = c.get("sub", 1)
    return make_dem(_domain(c, r), 0.1 if c["kind"] == "dem" else 1.0 / sub, _gravity(c), contact, r, mass, pos, vel,
                    omega=omega, periodic=_periodic(c), E=YOUNG, nu=POISSON, wall_E=YOUNG, wall_nu=POISSON, max_coord=16,
                    model="linear" if linear else "hertz",
                    freeze=np.ones(len(r), np.int32) if c["kind"] in ("bed", "grad") else None,
                    compat="wrapped" if c.get("wrapped") else "reference")


def prepare(case, seed):
    from lbdem_taichi_b200.lbdem.psclattice3d import PSCLattice3D
    from lbdem_taichi_b200.lbm3d.lattice import BasicLattice3D, ForcedLattice3D
    c = case
    s = dict(c=c, dem=None, lat=None)
    if c["kind"] == "fluid":
        args = (c["nx"], c["ny"], c["nz"], 1.0 / c["tau"], 1.0, 1.0, 1.0)
        lat = (ForcedLattice3D(*args, (1e-5, 0.0, 0.0), storage=c["storage"]) if c["cls"] == "forced" else
               BasicLattice3D(*args, storage=c["storage"]))
        lat.vel.from_numpy(_start_velocity(c, seed))
    else:
        s["dem"] = dem = _build_dem(c, seed)
        if c["kind"] == "dem":
            return s
        kw = dict(storage=c.get("storage", "f32"))
        if c["kind"] == "grad":
            kw.update(body_force=(2e-6, 0.0, 0.0), solid_fraction="smooth")
        elif c["kind"] != "bed":
            kw.update(smagorinsky=c.get("smag", "reference"), stress=c["kind"] == "shear",
                      lagged_storage="f16" if c.get("lag16") else None,
                      body_force=(FLUID_FORCE, 0.0, 0.0) if c.get("force") else None)
        lat = PSCLattice3D(c["nx"], c["ny"], c["nz"], 1.0 / c["tau"], 1.0, 1.0, 1.0, dem, **kw)
        if "cs" in c:
            lat.SmagorinskyConstant = c["cs"]
    ct = _cell_types(c)
    if ct is not None:
        lat.CT.from_numpy(ct)
    if c["kind"] == "bed":
        lat.vel[:, :, :, 0] = INLET_U
        lat.rho[c["nx"] - 1] = 1.0
    elif c["kind"] == "shear":
        lat.vel[:, :, 0, 0] = -WALL_U
        lat.vel[:, :, c["nz"] - 1, 0] = WALL_U
    lat.initialize()
    s["lat"] = lat
    if c["kind"] == "grad":
        from lbdem_taichi_b200.lbdem.adjoint import FrozenBedDrag
        s["problem"] = FrozenBedDrag(lat, c["steps"], (1.0, 0.0, 0.0), c["every"])
        s["F"] = torch.tensor([2e-6, 0.0, 0.0], dtype=torch.float64, device="cuda", requires_grad=True)
        s["P"] = torch.tensor(_inputs(c, seed)[0], dtype=torch.float64, device="cuda", requires_grad=True)
    return s


def run(state):
    c, lat, dem = state["c"], state["lat"], state["dem"]
    kind = c["kind"]
    if kind == "grad":
        from lbdem_taichi_b200.lbdem.adjoint import drag_loss
        state["F"].grad = state["P"].grad = None
        loss = drag_loss(state["F"], state["P"], state["problem"])
        loss.backward()
        return {"loss": loss.detach().float(), "force_grad": state["F"].grad.float(), "position_grad": state["P"].grad.float()}
    if kind == "dem":
        dem.run_substeps(c["sub"])
        t = dem._t
        return {k: t[k] for k in ("position", "velocity", "omega", "quaternion", "force", "moment")}
    if kind == "couple" and c["loop"] == "run":
        lat.run(c["steps"], c["sub"])
    else:
        for _ in range(c["steps"]):
            lat.collide()
            lat.stream()
            if kind == "shear":
                lat.compute_stress()
            if dem is not None:
                for _ in range(c.get("sub", 1)):
                    dem.run_simulation()
    out = {"f": lat._f[lat._cur]}
    if dem is not None:
        t = dem._t
        out["position"] = t["position"]
        out.update({k: t[k].float() for k in ("velocity", "omega", "force_fluid", "moment_fluid")})
    if kind == "shear":
        out["plane_stress"] = np.asarray(lat.compute_plane_average_stress(2, c["nz"] // 2), np.float32)
    return out


def work(case):
    c = case
    if c["kind"] == "dem":
        # positions, velocities, rotations, accelerations, contact histories in and out; contact law and integration
        return {"bytes": c["n"] * 2 * 8 * (3 * 9 + 4 + 3 * 10.0), "flops": c["n"] * c["sub"] * (3 * 400.0 + 300.0)}
    cells, es = float(c["nx"]) * c["ny"] * c["nz"], 4 if c.get("storage", "f32") == "f32" else 2
    if c["kind"] == "grad":
        # forward steps, and for each one step back: the state it read, the adjoint in and out
        return {"bytes": cells * c["steps"] * (2 * 76.0 + 3 * 76.0), "flops": cells * c["steps"] * 900.0}
    smag = c.get("smag", "reference") if c["kind"] in ("couple", "shear") else ("reference" if c.get("cls") == "basic" else "off")
    lag = 0.0 if smag != "reference" else 10.0 * (2 if c.get("lag16") else es)
    stress = 28.0 if c["kind"] == "shear" else 0.0
    return {"bytes": c["steps"] * cells * (38.0 * es + lag + stress),
            "flops": c["steps"] * cells * (330.0 if smag == "reference" else 250.0)}


# --------------------------------------------------------------------------------- 64-bit reference
def _f64(a, dev):
    return torch.as_tensor(np.asarray(a), dtype=torch.float64, device=dev)


class _Grains:
    """Spheres and their contacts at 64 bits: soft-sphere laws with shear history, improved Verlet."""

    def __init__(self, c, seed, dev):
        pos, r, vel, om, mass = _inputs(c, seed)
        self.c, self.dev, self.n = c, dev, len(r)
        self.pos, self.vel, self.om = _f64(pos, dev), _f64(vel, dev), _f64(om, dev)
        self.r, self.m = _f64(r, dev), _f64(mass, dev)
        z = torch.zeros_like(self.pos)
        self.acc, self.alpha, self.ff, self.mf, self.force, self.moment = z.clone(), z.clone(), z.clone(), z.clone(), z.clone(), z.clone()
        self.q = torch.zeros((self.n, 4), dtype=torch.float64, device=dev)
        self.q[:, 0] = 1.0
        self.dt = 0.1 if c["kind"] == "dem" else 1.0 / c.get("sub", 1)
        self.g = _f64(_gravity(c), dev)
        self.frozen = c["kind"] in ("bed", "grad")
        dom, per = _domain(c, r), _periodic(c)
        self.per, self.lo, self.hi = per, [dom[0], dom[2], dom[4]], [dom[1], dom[3], dom[5]]
        self.images = bool(c.get("wrapped"))
        self.linear = c["kind"] == "bed" or c.get("model") == "linear"
        self.i = None
        self.wshear = {a: torch.zeros((self.n, 3), dtype=torch.float64, device=dev) for a in range(6)}

    def candidates(self):
        """Pairs i < j whose surfaces may touch soon; the shear history of known ones is carried over."""
        i, j = [], []
        reach = 2.0 * float(self.r.max()) + 0.3
        for b in range(0, self.n, 1000):
            d = self._delta(self.pos[b:b + 1000, None, :], self.pos[None], self.images).norm(dim=-1)
            a, k = torch.nonzero(d < reach, as_tuple=True)
            keep = k > a + b
            i.append(a[keep] + b)
            j.append(k[keep])
        i, j = torch.cat(i), torch.cat(j)
        shear = torch.zeros((len(i), 3), dtype=torch.float64, device=self.dev)
        if self.i is not None and len(i) and len(self.i):
            old, new = self.i * self.n + self.j, i * self.n + j
            at = torch.searchsorted(old, new).clamp(max=len(old) - 1)
            same = old[at] == new
            shear[same] = self.shear[at[same]]
        o = torch.argsort(i * self.n + j)
        self.i, self.j, self.shear = i[o], j[o], shear[o]

    def _delta(self, a, b, image):
        d = b - a
        if image:
            for k in range(3):
                if self.per[k]:
                    L = self.hi[k] - self.lo[k]
                    d[..., k] -= L * torch.round(d[..., k] / L)
        return d

    @staticmethod
    def _frame(a):
        """Rows of the rotation that takes the unit vectors a onto +x about a x e_x."""
        x = torch.zeros_like(a)
        x[:, 0] = 1.0
        v = torch.linalg.cross(a, x)
        s2, co = (v * v).sum(1), a[:, 0]
        K = torch.zeros((len(a), 3, 3), dtype=a.dtype, device=a.device)
        K[:, 0, 1], K[:, 0, 2], K[:, 1, 2] = -v[:, 2], v[:, 1], -v[:, 0]
        K[:, 1, 0], K[:, 2, 0], K[:, 2, 1] = v[:, 2], -v[:, 1], v[:, 0]
        coef = torch.where(s2 > 1e-24, (1 - co) / s2.clamp(min=1e-300), torch.zeros_like(s2))
        E = torch.eye(3, dtype=a.dtype, device=a.device)
        R = E + K + coef[:, None, None] * (K @ K)
        flat = s2 <= 1e-24
        if bool(flat.any()):
            D = torch.diag_embed(torch.where(co[flat, None] > 0, torch.ones_like(a[flat]),
                                             a.new_tensor([-1.0, 1.0, -1.0]).expand(int(flat.sum()), 3)))
            R[flat] = D
        return R

    def _law(self, wall, Rs, ms, depth, vc, shear):
        if self.linear:
            kn, ks = (LIN_KN, LIN_KS) if wall else (LIN_KN / 2, LIN_KS / 2)
            kt = torch.full_like(depth, ks)
            gt = torch.zeros_like(depth)
            F0 = kn * depth - 2 * LIN_DN * torch.sqrt(kn * ms) * vc[:, 0]
            mu = LIN_MU
        else:
            Ys = YOUNG / (2 * (1 - POISSON ** 2))
            Gs = YOUNG / (4 * (2 - POISSON) * (1 + POISSON))
            le = math.log(RESTITUTION)
            beta = le / math.sqrt(le * le + math.pi ** 2)
            a = torch.sqrt(Rs * depth)
            F0 = 4 / 3 * Ys * a * depth + 2 * beta * torch.sqrt(5 / 6 * 2 * Ys * a * ms) * vc[:, 0]
            kt = 8 * Gs * a
            gt = -2 * beta * torch.sqrt(5 / 6 * kt * ms)
            mu = FRICTION
        inc = vc * self.dt
        inc[:, 0] = 0.0
        shear = shear + inc
        ts = -kt[:, None] * shear
        tl = ts.norm(dim=1)
        slide = (tl >= mu * F0) & (tl > 0)
        ratio = torch.where(slide, mu * F0 / tl.clamp(min=1e-300), torch.ones_like(tl))
        F = torch.where(slide[:, None], ts * ratio[:, None], ts - gt[:, None] * vc)
        shear = torch.stack([shear[:, 0], torch.where(slide, -F[:, 1] / kt, shear[:, 1]),
                             torch.where(slide, -F[:, 2] / kt, shear[:, 2])], 1)
        F[:, 0] = F0
        return F, shear

    def substep(self):
        F, M = torch.zeros_like(self.pos), torch.zeros_like(self.pos)
        i, j = self.i, self.j
        if len(i):
            d = self._delta(self.pos[i], self.pos[j], self.images)
            dist = d.norm(dim=1)
            depth = self.r[i] + self.r[j] - dist
            on = depth > 0
            self.shear[~on] = 0.0
            i, j, d, dist, depth = i[on], j[on], d[on], dist[on], depth[on]
            a = d / dist[:, None]
            R = self._frame(a)
            ri = a * (self.r[i] - depth)[:, None]
            rj = ri - d
            dv = self.vel[j] + torch.linalg.cross(self.om[j], rj) - self.vel[i] - torch.linalg.cross(self.om[i], ri)
            vc = (R @ dv[:, :, None])[:, :, 0]
            f, sh = self._law(False, 1 / (1 / self.r[i] + 1 / self.r[j]), 1 / (1 / self.m[i] + 1 / self.m[j]), depth, vc,
                              self.shear[on])
            self.shear[on] = sh
            fj = (R.transpose(1, 2) @ f[:, :, None])[:, :, 0]
            F.index_add_(0, i, -fj)
            F.index_add_(0, j, fj)
            M.index_add_(0, i, torch.linalg.cross(ri, -fj))
            M.index_add_(0, j, torch.linalg.cross(rj, fj))
        for w in range(6):
            ax, s = w // 2, 1.0 if w % 2 == 0 else -1.0
            if self.per[ax]:
                continue
            nrm = torch.zeros(3, dtype=torch.float64, device=self.dev)
            nrm[ax] = s
            depth = self.pos[:, ax] * s - (self.hi[ax] if s > 0 else -self.lo[ax]) + self.r
            on = torch.nonzero(depth >= 0, as_tuple=True)[0]
            self.wshear[w][depth < 0] = 0.0
            if not len(on):
                continue
            dp = depth[on]
            ri = (self.r[on] - dp)[:, None] * nrm
            R = self._frame(nrm.expand(len(on), 3).contiguous())
            vc = (R @ (-(torch.linalg.cross(self.om[on], ri) + self.vel[on]))[:, :, None])[:, :, 0]
            f, sh = self._law(True, self.r[on], self.m[on], dp, vc, self.wshear[w][on])
            self.wshear[w][on] = sh
            fi = -(R.transpose(1, 2) @ f[:, :, None])[:, :, 0]
            F[on] += fi
            M[on] += torch.linalg.cross(ri, fi)
        self.force = F + self.m[:, None] * self.g + self.ff
        self.moment = M + self.mf
        if self.frozen:
            return
        dt = self.dt
        acc = self.force / self.m[:, None]
        self.vel = self.vel + 0.5 * (self.acc + acc) * dt
        self.pos = self.pos + self.vel * dt + 0.5 * acc * dt * dt
        for k in range(3):
            if self.per[k]:
                L, p = self.hi[k] - self.lo[k], self.pos[:, k]
                self.pos[:, k] = torch.where(p > self.hi[k], p - L, torch.where(p < self.lo[k], p + L, p))
        self.acc = acc
        alpha = self.moment / (0.4 * self.m * self.r ** 2)[:, None]
        self.om = self.om + 0.5 * (self.alpha + alpha) * dt
        self.alpha = alpha
        q, w = self.q, self.om
        dq = 0.5 * torch.stack([-(q[:, 1] * w[:, 0] + q[:, 2] * w[:, 1] + q[:, 3] * w[:, 2]),
                                q[:, 0] * w[:, 0] - q[:, 3] * w[:, 1] + q[:, 2] * w[:, 2],
                                q[:, 3] * w[:, 0] + q[:, 0] * w[:, 1] + q[:, 1] * w[:, 2],
                                -q[:, 2] * w[:, 0] + q[:, 1] * w[:, 1] + q[:, 0] * w[:, 2]], 1)
        q = q + dq * dt
        self.q = q / q.norm(dim=1, keepdim=True)

    # ---- mapping onto the lattice: owner and solid fraction of every cell (nz, ny, nx)
    def shapes(self):
        """Sphere copies to map: (owner, centre in lattice units); the periodic images in wrapped mode."""
        p = self.pos + 0.5
        own = torch.arange(self.n, device=self.dev)
        if self.images:
            size = (self.c["nx"], self.c["ny"], self.c["nz"])
            for k in range(3):
                if not self.per[k]:
                    continue
                L, reach = self.hi[k] - self.lo[k], self.r[own] - 0.5 + 0.8660254037844386
                low, high = p[:, k] - reach < 0, p[:, k] + reach > size[k] - 1
                high &= ~low
                sh = torch.zeros(3, dtype=torch.float64, device=self.dev)
                sh[k] = L
                own = torch.cat([own, own[low], own[high]])
                p = torch.cat([p, p[low] + sh, p[high] - sh])
        return own, p

    def solid(self, closed):
        """Owner id (-1: none) and solid fraction by 5^3 sub-samples; `closed`: cells the mapping leaves out."""
        c, dev = self.c, self.dev
        nx, ny, nz = c["nx"], c["ny"], c["nz"]
        best = torch.zeros(nx * ny * nz, dtype=torch.int64, device=dev)
        own, ctr = self.shapes()
        half = math.sqrt(3.0) / 2
        rmax = float(self.r.max()) - 0.5
        e = int(math.ceil(rmax + half)) + 1
        ax = torch.arange(-e, e + 1, device=dev)
        box = torch.stack(torch.meshgrid(ax, ax, ax, indexing="ij"), -1).reshape(-1, 3)
        off = -0.4 + 0.2 * torch.arange(5, dtype=torch.float64, device=dev)
        sub = torch.stack(torch.meshgrid(off, off, off, indexing="ij"), -1).reshape(-1, 3)
        step = max(1, 4_000_000 // len(box))
        for b in range(0, len(own), step):
            o, p = own[b:b + step], ctr[b:b + step]
            r = self.r[o] - 0.5
            cell = torch.round(p).long()[:, None, :] + box[None]
            d = (p[:, None, :] - cell).norm(dim=-1)
            inside = ((cell >= 0) & (cell < torch.tensor([nx, ny, nz], device=dev))).all(-1)
            at = (cell[..., 2] * ny + cell[..., 1]) * nx + cell[..., 0]
            near = inside & (d < r[:, None] + half) & (r > 0)[:, None]
            gi, ci = torch.nonzero(near, as_tuple=True)
            at, d = at[gi, ci], d[gi, ci]
            open_ = ~closed[at]
            gi, ci, at, d = gi[open_], ci[open_], at[open_], d[open_]
            full = d <= r[gi] - half
            cnt = torch.full_like(at, 125)
            part = torch.nonzero(~full, as_tuple=True)[0]
            for k in range(0, len(part), 1_000_000):
                w = part[k:k + 1_000_000]
                v = (p[gi[w]] - cell[gi[w], ci[w]])[:, None, :] - sub[None]
                cnt[w] = (v.norm(dim=-1) < r[gi[w], None]).sum(1)
            key = full.long() * (1 << 40) + cnt * (1 << 30) + ((1 << 30) - 1 - o[gi])
            key = torch.where(cnt > 0, key, torch.zeros_like(key))
            best.scatter_reduce_(0, at, key, "amax")
        gid = torch.where(best > 0, (1 << 30) - 1 - (best & ((1 << 30) - 1)), torch.full_like(best, -1))
        eps = torch.where(best >> 40 > 0, torch.ones_like(best, dtype=torch.float64), ((best >> 30) & 1023).double() / 125)
        return gid, eps

    def lever(self, cells, gid):
        """Lever arms of cells (flat index) about their owners' centres, minimum image in wrapped mode."""
        nx, ny = self.c["nx"], self.c["ny"]
        x = torch.stack([cells % nx, (cells // nx) % ny, cells // (nx * ny)], 1).double()
        return -self._delta(x, self.pos[gid] + 0.5, self.images)


def _feq(q, rho, u):
    cu = CQ[q][0] * u[0] + CQ[q][1] * u[1] + CQ[q][2] * u[2]
    return W[q] * ((rho - 1) + rho * (3 * cu + 4.5 * cu * cu - 1.5 * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2])))


def _moments(d):
    rho = 1 + sum(d)
    j = [sum(CQ[q][a] * d[q] for q in range(19) if CQ[q][a]) for a in range(3)]
    return rho, j


def _blocked(c, d, S):
    """Deviations d[q] (nz, ny, nx) as the device keeps them: S d / w in x-blocks of 32, padded with zeros."""
    nb = -(-c["nx"] // 32)
    h = torch.zeros((c["nz"] * c["ny"], nb * 32, 19), dtype=torch.float64, device=d[0].device)
    for q in range(19):
        h[:, :c["nx"], q] = (d[q] * (S / W[q])).reshape(c["nz"] * c["ny"], c["nx"])
    return h.reshape(-1, 32, 19).transpose(1, 2).contiguous()


class _Fluid:
    """D3Q19 populations as deviations from the weights, (nz, ny, nx) per direction, at 64 bits."""

    def __init__(self, c, dev, force=None, smag="off"):
        self.c, self.dev, self.force, self.smag = c, dev, force, smag
        shape = (c["nz"], c["ny"], c["nx"])
        ct = _cell_types(c)
        if ct is not None:
            self.ct = torch.as_tensor(np.ascontiguousarray(ct.transpose(2, 1, 0)), device=dev)
        else:
            self.ct = torch.full(shape, FLUID, dtype=torch.int32, device=dev)
        self.om0 = 1.0 / c["tau"]
        z = torch.zeros(shape, dtype=torch.float64, device=dev)
        self.u0 = [z.clone(), z.clone(), z.clone()]
        self.wall = (self.ct == OBSTACLE) | (self.ct == MOVING)
        self.lag = None

    def start(self):
        one = torch.ones_like(self.u0[0])
        self.d = [torch.where(self.wall, -W[q] * one, _feq(q, one, self.u0)) for q in range(19)]
        self.lag = [one.clone(), *(torch.where(self.wall, 0 * u, u) for u in self.u0), self.om0 * one]
        self.rho = one.clone()
        self.pending = False

    def stream(self):
        """Pull; bounce-back at walls, with the wall's momentum where it moves; open x faces left to open_faces()."""
        src, ct = self.d, self.ct
        new = []
        for q in range(19):
            cx, cy, cz = CQ[q]
            v = torch.roll(src[q], (cz, cy, cx), (0, 1, 2))
            if q:
                n = torch.roll(ct, (cz, cy, cx), (0, 1, 2))
                solid = (n == OBSTACLE) | (n == MOVING) | (n == INLET_LEFT)
                back = src[OPP[q]]
                if self.c["kind"] in ("shear", "bed"):
                    cu = sum(k * torch.roll(u, (cz, cy, cx), (0, 1, 2)) for k, u in zip((cx, cy, cz), self.u0) if k)
                    r = torch.where(n == INLET_LEFT, torch.roll(self.rho, (cz, cy, cx), (0, 1, 2)), self.rho)
                    back = torch.where((n == MOVING) | (n == INLET_LEFT), back + 6 * W[q] * r * cu, back)
                v = torch.where(solid, back, v)
            new.append(torch.where(self.wall, src[q], v))
        return new

    def open_faces(self, d):
        """Zou-He pressure outlet (rho = 1) at the last x plane; the inlet plane keeps its populations and takes its
        neighbour's density.  Returns the outlet's normal velocity."""
        for q in range(19):
            d[q][..., 0] = self.d[q][..., 0]
        K = sum(d[q][..., -1] for q in range(19) if CQ[q][0] == 0)
        O = sum(d[q][..., -1] for q in range(19) if CQ[q][0] == 1)
        un = K + 2 * O      # u = -(rho - 1 - K - 2 O) / rho with rho = 1
        Ny = 0.5 * sum(CQ[q][1] * d[q][..., -1] for q in range(19) if CQ[q][0] == 0)
        Nz = 0.5 * sum(CQ[q][2] * d[q][..., -1] for q in range(19) if CQ[q][0] == 0)
        for q in range(19):
            if CQ[q][0] == -1:
                d[q][..., -1] = (d[OPP[q]][..., -1] + 6 * W[q] * (-un)
                                 - 36 * W[q] * (CQ[q][1] * Ny + CQ[q][2] * Nz))
        return un

    def second(self, d):
        """sum_q c_a c_b d_q for xx, yy, zz, xy, xz, yz."""
        return [sum(CQ[q][a] * CQ[q][b] * d[q] for q in range(19) if CQ[q][a] * CQ[q][b])
                for a, b in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))]

    def noneq(self, d, rho, u):
        s = self.second(d)
        e = (rho - 1) / 3
        return [s[0] - e - rho * u[0] * u[0], s[1] - e - rho * u[1] * u[1], s[2] - e - rho * u[2] * u[2],
                s[3] - rho * u[0] * u[1], s[4] - rho * u[0] * u[2], s[5] - rho * u[1] * u[2]]

    def stress(self):
        """Plane average (xy, xz, yz) of the post-stream stress at z = nz // 2."""
        d = self.stream()
        P = self.noneq(d, self.lag[0], self.lag[1:4])
        k = -(1 - 0.5 * self.lag[4])
        z = self.c["nz"] // 2
        return np.array([float((k * P[m])[z].mean()) for m in (3, 4, 5)])

    def step(self, grains=None):
        """One collide (of the streamed state, but for the first); grains get their force and torque."""
        bed = self.c["kind"] == "bed"
        d = self.stream() if self.pending else self.d
        un = None
        if bed and self.pending:
            un = self.open_faces(d)
        self.pending = True
        rho, j = _moments(d)
        u = [x / rho for x in j]
        if bed:
            rho[..., -1] = 1.0
            u[0][..., -1] = un if un is not None else INLET_U
            u[1][..., -1] = u[2][..., -1] = 0.0
            if un is not None:
                rho[..., 0] = rho[..., 1]
            else:
                rho[..., 0] = 1.0
        om = torch.full_like(rho, self.om0)
        if self.smag != "off":
            P = self.noneq(d, *((self.lag[0], self.lag[1:4]) if self.smag == "reference" else (rho, u)))
            rate = torch.sqrt(2 * (P[0] ** 2 + P[1] ** 2 + P[2] ** 2) + 4 * (P[3] ** 2 + P[4] ** 2 + P[5] ** 2))
            prev = self.lag[4] if self.smag == "reference" else self.om0
            om = 1 / (1 / self.om0 + 4.5 * self.c.get("cs", 0.1) ** 2 * prev * rate / rho)
        self.lag = [rho, *u, om]
        self.rho = rho
        B = us = None
        if grains is not None:
            closed = (self.wall if not bed else torch.zeros_like(self.wall)).reshape(-1)
            gid, eps = grains.solid(closed)
            cells = torch.nonzero(gid >= 0, as_tuple=True)[0]
            g, e = gid[cells], eps[cells]
            t = 1 / om.reshape(-1)[cells] - 0.5
            b = e * t / ((1 - e) + t)
            r = grains.lever(cells, g)
            v = grains.vel[g] + torch.linalg.cross(grains.om[g], r)
            h = b[:, None] * (torch.stack([x.reshape(-1)[cells] for x in j], 1) - rho.reshape(-1)[cells, None] * v)
            grains.ff = torch.zeros_like(grains.pos).index_add_(0, g, h)
            grains.mf = torch.zeros_like(grains.pos).index_add_(0, g, torch.linalg.cross(r, h))
            B = torch.zeros_like(rho)
            B.view(-1)[cells] = b
            us = []
            for a in range(3):
                w = torch.zeros_like(rho)
                w.view(-1)[cells] = v[:, a]
                us.append(w)
        new = []
        for q in range(19):
            fe = _feq(q, rho, u)
            x = -om * (d[q] - fe)
            if B is not None:
                x = (1 - B) * x + B * (d[OPP[q]] - _feq(OPP[q], rho, u) + _feq(q, rho, us) - d[q])
            x = d[q] + x
            if self.force is not None:
                x = x + 3 * W[q] * rho * sum(CQ[q][a] * self.force[a] for a in range(3))
            keep = self.wall
            if bed:
                keep = keep | (self.ct == INLET_LEFT)
            new.append(torch.where(keep, self.d[q], x))
        self.d = new


def _exact_grad(c, seed, dev):
    """Drag on the bed and its gradients by automatic differentiation of the same steps."""
    from torch.utils.checkpoint import checkpoint
    F = torch.tensor([2e-6, 0.0, 0.0], dtype=torch.float64, device=dev, requires_grad=True)
    pos, r = _inputs(c, seed)[:2]
    P = _f64(pos, dev).requires_grad_(True)
    r = _f64(r, dev) - 0.5
    fl = _Fluid(c, dev)
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    # owner of each cell: the largest smooth fraction; one cell belongs to one sphere's ramp here or the lowest id
    e = int(math.ceil(float(r.max()) + 0.5)) + 1
    ax = torch.arange(-e, e + 1, device=dev)
    box = torch.stack(torch.meshgrid(ax, ax, ax, indexing="ij"), -1).reshape(-1, 3)
    ctr = P.detach() + 0.5
    best = torch.zeros(nx * ny * nz, dtype=torch.float64, device=dev)
    cell = torch.round(ctr).long()[:, None, :] + box[None]
    inside = ((cell >= 0) & (cell < torch.tensor([nx, ny, nz], device=dev))).all(-1)
    t = (r[:, None] - (ctr[:, None, :] - cell).norm(dim=-1) + 0.5).clamp(0, 1)
    eps = torch.where(inside, t * t * (3 - 2 * t), torch.zeros_like(t))
    at = ((cell[..., 2] * ny + cell[..., 1]) * nx + cell[..., 0]).clamp(0, nx * ny * nz - 1)
    eps = torch.where(fl.wall.reshape(-1)[at], torch.zeros_like(eps), eps)
    best.scatter_reduce_(0, at.reshape(-1), eps.reshape(-1), "amax")
    mine = (eps > 0) & (eps == best[at])
    owner = torch.full((nx * ny * nz,), len(r), dtype=torch.int64, device=dev)
    g, k = torch.nonzero(mine, as_tuple=True)
    owner.scatter_reduce_(0, at[g, k], g, "amin")
    cells = torch.nonzero(owner < len(r), as_tuple=True)[0]
    g = owner[cells]
    x = torch.stack([cells % nx, (cells // nx) % ny, cells // (nx * ny)], 1).double()
    t = (r[g] - (P[g] + 0.5 - x).norm(dim=1) + 0.5).clamp(max=1.0)
    ep = t * t * (3 - 2 * t)
    tm = c["tau"] - 0.5
    B = torch.zeros(nx * ny * nz, dtype=torch.float64, device=dev).index_put((cells,), ep * tm / ((1 - ep) + tm)).reshape(nz, ny, nx)
    om, wall, ct = fl.om0, fl.wall, fl.ct
    solid = []
    for q in range(19):
        cx, cy, cz = CQ[q]
        solid.append(torch.roll(ct, (cz, cy, cx), (0, 1, 2)) == OBSTACLE)

    def collide(d, B, F):
        rho, j = _moments(d)
        u = [v / rho for v in j]
        z = torch.zeros_like(rho)
        fe = [_feq(q, rho, u) for q in range(19)]
        out = []
        for q in range(19):
            v = d[q] - (1 - B) * om * (d[q] - fe[q]) + B * (d[OPP[q]] - fe[OPP[q]] + W[q] * (rho - 1) - d[q])
            v = v + 3 * W[q] * rho * sum(CQ[q][a] * F[a] for a in range(3) if CQ[q][a]) if q else v
            out.append(torch.where(wall, d[q], v))
        return out, (B * j[0] + z).sum()

    def one(first, d, B, F):
        d = list(torch.unbind(d))
        if not first:
            new = []
            for q in range(19):
                cx, cy, cz = CQ[q]
                v = torch.roll(d[q], (cz, cy, cx), (0, 1, 2))
                v = torch.where(solid[q], d[OPP[q]], v) if q else v
                new.append(torch.where(wall, d[q], v))
            d = new
        out, drag = collide(d, B, F)
        return torch.stack(out), drag

    fl.start()
    d = torch.stack(fl.d)
    for s in range(c["steps"]):
        d, drag = checkpoint(one, s == 0, d, B, F, use_reentrant=False)
    drag.backward()
    return {"loss": drag.detach(), "force_grad": F.grad, "position_grad": P.grad}


def exact(case, seed):
    c = case
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    with torch.no_grad():
        if c["kind"] == "dem":
            g = _Grains(c, seed, dev)
            g.candidates()
            for _ in range(c["sub"]):
                g.substep()
            return {"position": g.pos, "velocity": g.vel, "omega": g.om, "quaternion": g.q, "force": g.force, "moment": g.moment}
        if c["kind"] != "grad":
            cells = c["nx"] * c["ny"] * c["nz"]
            grains = None
            if c["kind"] == "fluid":
                fl = _Fluid(c, dev, (1e-5, 0.0, 0.0) if c["cls"] == "forced" else None, "off" if c["cls"] == "forced" else "reference")
                v = _start_velocity(c, seed)
                fl.u0 = [_f64(np.ascontiguousarray(v[..., a].transpose(2, 1, 0)), dev) for a in range(3)]
            else:
                grains = _Grains(c, seed, dev)
                smag = "off" if c["kind"] == "bed" else c.get("smag", "reference")
                fl = _Fluid(c, dev, (FLUID_FORCE, 0.0, 0.0) if c.get("force") else None, smag)
                if c["kind"] == "bed":
                    fl.u0[0][:] = INLET_U
                elif c["kind"] == "shear":
                    fl.u0[0][0], fl.u0[0][-1] = -WALL_U, WALL_U
            if dev == "cpu" and cells > 200_000:
                return None
            fl.start()
            stress = None
            for s in range(c["steps"]):
                fl.step(grains)
                if c["kind"] == "shear" and s == c["steps"] - 1:
                    stress = fl.stress()
                if grains is not None:
                    grains.candidates()
                    for _ in range(c.get("sub", 1)):
                        grains.substep()
            S = SCALE[c["storage"]]
            out = {"f": _blocked(c, fl.d, S)}
            if grains is not None:
                out.update(position=grains.pos, velocity=grains.vel, omega=grains.om, force_fluid=grains.ff,
                           moment_fluid=grains.mf)
            if stress is not None:
                out["plane_stress"] = stress
            return out
    return _exact_grad(c, seed, dev)
