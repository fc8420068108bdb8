"""The work whose speed this package answers for, as a list of measurable cases.

Each case is one of six uses of the public interface (windtunnel_b200.LBM and
its neighbours), at sizes from the interactive tunnel to the benchmark channels:

* ``channel``  a batch of steps (the pool's step(n)), then the flow fields
* ``frame``    one turn of the interactive loop: single steps with the force
               read after each, the slice view, a smoke-particle update
* ``design``   the drag of a solid-fraction field and its gradient, through
               torch autograd
* ``adjoint``  the same through LBM.adjoint, the lattice-sized form
* ``voxel``    a triangle mesh made into an occupancy grid
* ``place``    a voxel body moved in the lattice (the yaw / position sliders)

`prepare` sets a lattice up as a program does before its time loop (lattice,
parameters, body, seeded initial state), `run` is one pass of the loop,
`exact` the same numbers from a plain float64 torch lattice in this file.
"""
from __future__ import annotations

import math

import numpy as np
import torch
import torch.utils.checkpoint

from windtunnel_b200 import LBM
from windtunnel_b200.autograd import drag
from windtunnel_b200.bodies import body_box, body_matrix, superellipsoid_grid
from windtunnel_b200.mesh import hull_mesh, orient, voxel_build

ELEM = {"f32": 4, "f16dev": 2, "f64": 8}
HULL = dict(semi=(0.5, 0.1875, 0.15), exponent=2.5)

# float operations of one cell update (collision of 19 populations with the
# eddy viscosity and two relaxation rates), and of its vector-Jacobian product
FLOPS_STEP, FLOPS_VJP = 320, 800


def _lattice(name, kind, dims, storage="f32", math_="fast", side="eq", rounding="nearest",
             body="hull", ground=False, road=0.0, les=True, trt=True, u0=0.06, tau=0.5072, steps=100,
             **more):
    c = dict(kind=kind, nx=dims[0], ny=dims[1], nz=dims[2], storage=storage, math=math_, side=side,
             rounding=rounding, body=body, ground=ground, road=road, les=les, trt=trt, u0=u0,
             tau=tau, steps=steps, **more)
    return dict(c, name=name) if name else c


def listed():
    return [
        # The interactive tunnel on its smallest grid: latency and launches.
        _lattice("frame_small", "frame", (64, 32, 32), body="sphere", tau=0.515, steps=4,
                 particles=2000),
        # The validation page: a car on the road, the reference's own arithmetic
        # bit for bit, its averaging window in one batch.
        _lattice("validate_exact", "channel", (96, 44, 44), math_="exact", body="car", ground=True,
                 tau=0.503, steps=300),
        # A car over a rolling road with turning wheels (moving walls). Such
        # runs compare drag to a percent, so they are made in float32.
        _lattice("road_f32", "channel", (160, 80, 80), body="car", ground=True, road=0.06,
                 tau=0.515, steps=100),
        # A lattice fitted to a body with no regard to round numbers.
        _lattice("ragged_f32", "channel", (193, 85, 91), body="sphere", tau=0.515, steps=100),
        # The benchmark channel in float32 storage, free-slip sides.
        _lattice("channel256_f32", "channel", (256, 128, 128), side="freeslip", steps=200),
        # The same in half storage with the rounding that keeps Cd.
        _lattice("channel256_f16sr", "channel", (256, 128, 128), storage="f16dev", side="freeslip",
                 rounding="stochastic", tau=0.515, steps=150),
        # The largest configuration: half storage, nearest rounding.
        _lattice("channel512_f16", "channel", (512, 192, 192), storage="f16dev", side="freeslip",
                 steps=300),
        # The float64 form the other forms are judged by.
        _lattice("oracle_f64", "channel", (192, 96, 96), storage="f64", side="freeslip", steps=100),
        # One gradient of a shape-optimisation loop, through autograd.
        _lattice("design_f32", "design", (128, 64, 64), side="freeslip", body="none", u0=0.05,
                 tau=0.524, steps=150, window=50, checkpoint=50, half=16),
        # The gradient at scale: half forward states, square-root checkpoints.
        _lattice("adjoint_f16", "adjoint", (384, 160, 160), storage="f16dev", side="freeslip",
                 body="none", tau=0.5072, steps=64, window=16, checkpoint=8, half=32),
        # A 20000-triangle mesh loaded at the benchmark's resolution.
        dict(name="voxel_hull", kind="voxel", nu=100, nv=100, res=160),
        # The voxel body turned in the benchmark channel.
        _lattice("place_hull", "place", (256, 128, 128), side="freeslip", steps=0, res=160),
    ]


def _dims(rng, lo, hi, even):
    """Dimensions of lo..hi cells in all, spread over their logarithm: a channel
    about twice as long as wide."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    w = (n / 2.2) ** (1 / 3)
    ny, nz = (max(12, round(w * rng.uniform(0.85, 1.15))) for _ in range(2))
    nx = max(16, round(n / (ny * nz)))
    return (nx + nx % 2 if even else nx | 1), ny, nz


def draw(rng):
    kind = rng.choice(["channel"] * 6 + ["frame", "design", "adjoint", "voxel", "place"])
    # runs short and viscous enough that two roundings of one flow stay
    # comparable: at lower viscosity the wake amplifies them
    tau = round(rng.uniform(0.512, 0.53), 4)
    side = rng.choice(["eq", "freeslip"])
    if kind == "voxel":
        return dict(kind=kind, nu=rng.randint(20, 110), nv=rng.randint(20, 110),
                    res=rng.randint(48, 176))
    if kind == "frame":
        return _lattice(None, kind, _dims(rng, 2e4, 5e5, rng.random() < 0.7), body="sphere",
                        side=side, tau=tau, steps=rng.randint(1, 8),
                        particles=int(math.exp(rng.uniform(math.log(200), math.log(20000)))))
    if kind == "place":
        return _lattice(None, kind, _dims(rng, 1e5, 6e6, rng.random() < 0.7),
                        storage=rng.choice(["f32", "f16dev"]), side=side, steps=0,
                        res=rng.randint(64, 160))
    if kind in ("design", "adjoint"):
        storage = "f32" if kind == "design" else rng.choice(["f32", "f16dev"])
        dims = _dims(rng, 6e4, 6e5 if kind == "design" else 4e6, rng.random() < 0.7)
        steps = rng.randint(24, 64)
        return _lattice(None, kind, dims, storage=storage, side=side, body="none", tau=tau,
                        steps=steps, window=rng.randint(1, steps // 2),
                        checkpoint=rng.choice([0, 8, 13]), half=min(dims) // 4)
    form = rng.choice(["f32", "f32", "road", "f16dev", "f16sr", "exact", "f64"])
    even = rng.random() < 0.7
    les, trt = rng.choice([(True, True), (True, True), (True, False), (False, True)])
    more = dict(tau=tau if les else max(tau, 0.52), les=les, trt=trt, steps=rng.randint(40, 120))
    if form == "road":
        return _lattice(None, kind, _dims(rng, 5e4, 5e6, even), body="car", ground=True, road=0.06,
                        **more)
    big = 2e6 if form in ("exact", "f64") else 8e6
    return _lattice(None, kind, _dims(rng, 3e4, big, even), side=side,
                    storage={"f16sr": "f16dev", "exact": "f32"}.get(form, form),
                    math_="exact" if form == "exact" else "fast",
                    rounding="stochastic" if form == "f16sr" else "nearest",
                    body=rng.choice(["hull", "sphere", "car"]), ground=rng.random() < 0.3, **more)


# ---- bodies ---------------------------------------------------------------------------

def _placed(case, seed):
    """Yaw and position of the body, a little different for every seed."""
    r = np.random.default_rng(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    yaw = math.radians(15.0 + r.uniform(-4, 4))
    return yaw, [0.36 * nx + r.uniform(-0.5, 0.5), 0.5 * ny + r.uniform(-0.5, 0.5),
                 0.5 * nz + r.uniform(-0.5, 0.5)]


def _body(case, seed):
    """Occupancy of the case's body: (x0, y0, z0) of a block of cells, its mask
    [z][y][x], and for turning wheels the cells' wall velocities."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    yaw, P = _placed(case, seed)
    kind = case["body"]
    size = min(0.31 * nx, 0.9 * ny, 0.9 * nz)
    if kind == "none":
        return (1, 1, 1), np.zeros((1, 1, 1), bool), None
    if kind == "sphere":
        r = 0.24 * size
        w = [r, r, r]
    elif kind == "hull":
        M = body_matrix(yaw, 0.0)
        b = body_box(M, HULL["semi"], size, P)
        w = [(b[k + "1"] - b[k + "0"]) / 2 for k in "xyz"]
    else:
        P[1] = 1.0
        w = [0.5 * size, 0.34 * size, 0.22 * size]
    lo = [max(1, int(math.floor(P[k] - w[k]))) for k in range(3)]
    hi = [min((nx, ny, nz)[k] - 2, int(math.ceil(P[k] + w[k]))) for k in range(3)]
    z, y, x = (np.arange(lo[k], hi[k] + 1) + 0.5 for k in (2, 1, 0))
    dx, dy, dz = x[None, None, :] - P[0], y[None, :, None] - P[1], z[:, None, None] - P[2]
    wheels = None
    if kind == "sphere":
        mask = dx * dx + dy * dy + dz * dz <= r * r
    elif kind == "hull":
        a = (M[0] * dx + M[3] * dy + M[6] * dz) / size
        b = (M[1] * dx + M[4] * dy + M[7] * dz) / size
        c = (M[2] * dx + M[5] * dy + M[8] * dz) / size
        e = HULL["exponent"]
        mask = sum(np.abs(v / s) ** e for v, s in zip((a, b, c), HULL["semi"])) <= 1
    else:
        X, Y, Z = dx / size, dy / size, dz / size
        mask = (np.abs(X) <= 0.45) & (np.abs(Y - 0.13) <= 0.06) & (np.abs(Z) <= 0.18)
        mask |= ((X - 0.03) / 0.26) ** 2 + ((Y - 0.19) / 0.12) ** 2 + (Z / 0.16) ** 2 <= 1
        spin = np.zeros(mask.shape + (3,))
        turning = np.zeros(mask.shape, bool)
        for cx in (-0.29, 0.28):
            wheel = ((X - cx) ** 2 + (Y - 0.075) ** 2 <= 0.075 ** 2) & \
                (np.abs(np.abs(Z) - 0.17) <= 0.04)
            mask |= wheel
            if case["road"]:
                om = case["road"] / 0.075
                spin[..., 0] = np.where(wheel, om * (0.075 - Y), spin[..., 0])
                spin[..., 1] = np.where(wheel, om * (X - cx), spin[..., 1])
                turning |= wheel
        wheels = (turning, spin) if case["road"] else None
    return tuple(lo), np.broadcast_to(mask, (z.size, y.size, x.size)), wheels


def _fraction(case, seed):
    """Design box around (0.31 nx, ny/2, nz/2) and its solid fraction: a smoothed
    sphere plus noise."""
    h = case["half"]
    c = [round(0.31 * case["nx"]), case["ny"] // 2, case["nz"] // 2]
    c = [min(max(v, h + 1), n - h - 1) for v, n in zip(c, (case["nx"], case["ny"], case["nz"]))]
    box = tuple(v - h for v in c) + tuple(v + h for v in c)
    z, y, x = np.meshgrid(*[np.arange(2 * h) + 0.5 - h] * 3, indexing="ij")
    r = np.sqrt(x * x + y * y + z * z)
    s = 0.5 * (1 - np.tanh((r - 0.62 * h) / 1.5))
    s = s + np.random.default_rng(seed).uniform(-0.05, 0.05, s.shape)
    return box, np.clip(s, 0, 1)


# ---- the public calls -------------------------------------------------------------------

def _sim(case, seed):
    sim = LBM(case["nx"], case["ny"], case["nz"], storage=case["storage"], math=case["math"],
              side_bc=case["side"])
    sim.set_params(u0=case["u0"], tau=case["tau"], csm=0.1, les=int(case["les"]),
                   trt=int(case["trt"]), f16_rounding=case["rounding"], **{"lambda": 3 / 16})
    (x0, y0, z0), mask, wheels = _body(case, seed)
    ez, ey, ex = mask.shape
    box = (x0, y0, z0, x0 + ex - 1, y0 + ey - 1, z0 + ez - 1)
    if mask.any() or case["ground"]:
        sim.voxelize_mask(box, mask, case["ground"], wheels[0] if wheels else None,
                          wheels[1] if wheels else None, case["road"])
    sim.init_eq_noise(seed, 1e-4)
    return sim


def prepare(case, seed):
    kind = case["kind"]
    if kind == "voxel":
        tris = hull_mesh(nu=case["nu"], nv=case["nv"], seed=seed, **HULL)
        orient(tris, 0, 1)
        # one size for every seed: the bumps change, the bounds do not
        v = tris.reshape(-1, 3)
        v *= (np.array([1.0, 0.377, 0.303]) / (v.max(0) - v.min(0))).astype(np.float32)
        return dict(case=case, tris=tris)
    if kind == "place":
        sim = _sim(dict(case, body="none"), seed)
        grid = superellipsoid_grid(res=case["res"], **HULL)
        yaw, P = _placed(case, seed)
        return dict(case=case, sim=sim, grid=grid, yaw=yaw, P=P, turn=0,
                    scale=min(0.31 * case["nx"], 0.9 * case["ny"], 0.9 * case["nz"]))
    st = dict(case=case, sim=_sim(case, seed))
    if kind in ("design", "adjoint"):
        box, s = _fraction(case, seed)
        st.update(box=box, s=torch.tensor(s, dtype=torch.float32, requires_grad=True), s64=s)
    if kind == "frame":
        st["xyz"] = _particles(case, seed)
    return st


def _force_type(case):
    """The force series is kept in the type of the arithmetic that made it."""
    return np.float64 if case["math"] == "exact" or case["storage"] == "f64" else np.float32


def run(st):
    case, kind = st["case"], st["case"]["kind"]
    if kind == "voxel":
        g = voxel_build(st["tris"], case["res"])
        return dict(grid=g.grid, solid=g.solid, openness=g.openness)
    sim = st["sim"]
    if kind == "channel":
        forces = sim.step_forces(case["steps"])
        ux, uy, uz, rho = sim.fields()
        return dict(forces=forces.astype(_force_type(case)), ux=ux, uy=uy, uz=uz, rho=rho)
    if kind == "frame":
        forces = []
        for _ in range(case["steps"]):
            sim.step()
            forces.append(sim.force)
        view = sim.slice("xy", None, "speed")
        xyz, expired, speed = sim.advect(st["xyz"], 2.0)
        # a renderer's vertex buffer is float32
        return dict(forces=np.array(forces, np.float32), view=view, xyz=xyz.astype(np.float32),
                    expired=expired, speed=speed)
    if kind == "design":
        s = st["s"]
        s.grad = None
        J = drag(s, sim, st["box"], case["steps"], case["window"], 0, case["checkpoint"],
                 True).float()
        J.backward()
        return dict(J=J.detach(), grad=s.grad)
    if kind == "adjoint":
        # the design variables of an optimiser are float32, and so is their gradient
        sim.set_solid_fraction(st["box"], st["s64"])
        J, g, _ = sim.adjoint(case["steps"], case["window"], 0, case["checkpoint"], keep=True)
        return dict(J=np.float32(J), grad=g.astype(np.float32))
    st["turn"] += 1
    yaw = st["yaw"] + 0.05 * (st["turn"] % 7)
    M, g = body_matrix(yaw, 0.0), st["grid"]
    sim.voxelize_grid(g.grid, g.min, g.inv, M, st["P"], st["scale"],
                      body_box(M, g.ext, st["scale"], st["P"]))
    return dict(solid=sim.solid, frontal=sim.frontalArea, planform=sim.planformArea,
                cells=sim.solidCells, ride=sim.rideHeight)


def work(case):
    kind = case["kind"]
    if kind == "voxel":
        tris = 2 * case["nu"] * case["nv"]
        r = case["res"]
        cells = (r + 4) * (0.42 * r + 4) * (0.34 * r + 4)
        return dict(bytes=36 * tris + cells, flops=3 * 40 * tris * 4 + 60 * tris * 16)
    n = case["nx"] * case["ny"] * case["nz"]
    state = 19 * ELEM[case["storage"]] * n
    if kind == "place":
        return dict(bytes=3 * n, flops=40 * n * 0.02)
    if kind in ("design", "adjoint"):
        # forward and recomputed steps, then a backward step that reads the
        # state and the next adjoint and writes its own
        steps, adj = case["steps"], 19 * 4 * n
        return dict(bytes=steps * (2 * 2 * state + state + 2 * adj),
                    flops=steps * n * (2 * FLOPS_STEP + FLOPS_VJP))
    views = 16 * n if kind == "channel" else 12 * case["nx"] * case["ny"] + 200 * case["particles"]
    return dict(bytes=case["steps"] * 2 * state + views, flops=case["steps"] * n * FLOPS_STEP)


# ---- the same in float64 torch ------------------------------------------------------------
_E = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0),
      (-1, -1, 0), (1, -1, 0), (-1, 1, 0), (1, 0, 1), (-1, 0, -1), (1, 0, -1), (-1, 0, 1),
      (0, 1, 1), (0, -1, -1), (0, 1, -1), (0, -1, 1)]
_W = [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12
_AT = {e: q for q, e in enumerate(_E)}
_OPP = [_AT[(-a, -b, -c)] for a, b, c in _E]
_MY = [_AT[(a, -b, c)] for a, b, c in _E]
_MZ = [_AT[(a, b, -c)] for a, b, c in _E]


def _uniform(seed, k):
    """Draw k (an array) of the splitmix64 stream of the seeded initial state."""
    with np.errstate(over="ignore"):
        z = np.uint64(seed) + (k + np.uint64(1)) * np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    z = z ^ (z >> np.uint64(31))
    return (z >> np.uint64(11)).astype(np.float64) * 2.0 ** -53


def _equilibrium(rho, ux, uy, uz):
    usq = 1.5 * (ux * ux + uy * uy + uz * uz)
    out = []
    for (a, b, c), w in zip(_E, _W):
        cu = 3 * (a * ux + b * uy + c * uz)
        out.append(w * ((rho - 1) + rho * (cu + 0.5 * cu * cu - usq)))
    return torch.stack(out)


class _Exact:
    """The lattice in float64: populations f[q][z][y][x] as deviations."""

    def __init__(self, case, seed):
        self.case, dev = case, "cuda" if torch.cuda.is_available() else "cpu"
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        obj = np.zeros((nz, ny, nx), bool)
        (x0, y0, z0), mask, wheels = _body(case, seed)
        ez, ey, ex = mask.shape
        at = (slice(z0, z0 + ez), slice(y0, y0 + ey), slice(x0, x0 + ex))
        obj[at] = mask
        wall = np.zeros_like(obj)
        wall[:, 0, :] = case["ground"]
        vel = np.zeros((3, nz, ny, nx), np.float32)
        vel[0, :, 0, :] = case["road"]
        if wheels:
            for k in range(3):
                vel[k][at] = np.where(wheels[0] & mask, wheels[1][..., k], vel[k][at])
        T = lambda v: torch.as_tensor(v, device=dev)  # noqa: E731
        self.obj, self.solid = T(obj), T(obj | wall)
        inner = torch.zeros_like(self.obj)
        inner[1:-1, 1:-1, 1:-1] = True
        self.fluid = inner & ~self.solid
        self.links, self.corr = {}, {}
        vel = T(vel.astype(np.float64))
        moving = bool(case["road"])
        for q in range(1, 19):
            src = self._pull(self.solid, q)
            self.links[q] = (self.fluid & src, self.fluid & self._pull(self.obj, q))
            if moving:
                cu = sum(e * self._pull(vel[k], q) for k, e in enumerate(_E[q]))
                self.corr[q] = 6 * _W[q] * cu
        i = np.arange(nx * ny * nz, dtype=np.uint64)
        noise = [T(1e-4 * (2 * _uniform(seed, np.uint64(3) * i + np.uint64(k)) - 1)
                   .reshape(nz, ny, nx)) for k in range(3)]
        free = (~self.solid).double()
        self.u = [(noise[0] + case["u0"]) * free, noise[1] * free, noise[2] * free]
        self.rho = torch.ones_like(free)
        self.f = _equilibrium(self.rho, *self.u)
        one = torch.ones((), dtype=torch.float64, device=dev)
        self.eq = _equilibrium(one, case["u0"] * one, 0 * one, 0 * one)[:, None, None, None]
        eq_cell = torch.zeros_like(self.obj)
        eq_cell[:, 0, :] = True
        eq_cell &= ~self.solid
        for s in ((0,), (-1,), (slice(None), -1), (slice(None), slice(None), 0)):
            eq_cell[s] = True
        self.eq_cell = eq_cell

    @staticmethod
    def _pull(a, q):
        x, y, z = _E[q]
        return torch.roll(a, (z, y, x), (-3, -2, -1)) if q else a

    def _sides(self, f):
        """Free-slip: the side planes as mirrors of the layers beside them."""
        f = f.clone()
        f[:, :, 0], f[:, :, -1] = f[_MY][:, :, 1], f[_MY][:, :, -2]
        f[:, 0], f[:, -1] = f[_MZ][:, 1], f[_MZ][:, -2]
        return f

    def advance(self, f, rho, sfrac=None, last=True):
        """One step: new populations, density, velocity and the force."""
        case = self.case
        src = self._sides(f) if case["side"] == "freeslip" else f
        p, force = [src[0]], [0.0, 0.0, 0.0]
        for q in range(1, 19):
            solid, body = self.links[q]
            back = f[_OPP[q]]
            corr = self.corr[q] * rho if self.corr else None
            if corr is not None:
                back = back + corr
            p.append(torch.where(solid, back, self._pull(src[q], q)))
            ex_ = torch.where(body, f[_OPP[q]] + back, 0.0).sum()
            for k in range(3):
                if _E[q][k]:
                    force[k] = force[k] - _E[q][k] * ex_
        p = torch.stack(p)
        r = 1 + p.sum(0)
        u = [sum(e[k] * p[q] for q, e in enumerate(_E) if e[k]) / r for k in range(3)]
        n = p - _equilibrium(r, *u)
        tau = torch.full_like(r, case["tau"])
        if case["les"]:
            P = [[sum(e[a] * e[b] * n[q] for q, e in enumerate(_E) if e[a] * e[b])
                  for b in range(a, 3)] for a in range(3)]
            q2 = P[0][0] ** 2 + P[1][0] ** 2 + P[2][0] ** 2 + \
                2 * (P[0][1] ** 2 + P[0][2] ** 2 + P[1][1] ** 2)
            mag = torch.sqrt(2 * q2 + 1e-300)   # a finite slope at zero
            tau = 0.5 * (tau + torch.sqrt(tau * tau + 18 * math.sqrt(2) * 0.01 * mag / r))
        om = 1 / tau
        omm = 1 / (0.5 + (3 / 16) / (tau - 0.5)) if case["trt"] else om
        no = n[_OPP]
        g = p - om * 0.5 * (n + no) - omm * 0.5 * (n - no)
        if sfrac is not None:
            d = g - p[_OPP]
            for k in range(3):
                force[k] = force[k] + (sfrac * sum(e[k] * d[q] for q, e in enumerate(_E)
                                                   if e[k])).sum()
            g = g - sfrac * d
        g = torch.where(self.fluid, g, torch.where(self.eq_cell, self.eq, f))
        g = torch.cat([g[..., :-1], g[..., -2:-1]], -1)
        if not last and not self.corr:
            return g, rho, None, force
        keep = self.solid & ~self.eq_cell
        u = [torch.where(self.fluid, v, torch.where(keep, 0.0, u0))
             for v, u0 in zip(u, (case["u0"], 0.0, 0.0))]
        r = torch.where(self.fluid, r, 1.0)
        copy = lambda v: torch.cat([v[..., :-1], v[..., -2:-1]], -1)  # noqa: E731
        return g, copy(r), [copy(v) for v in u], force

    def steps(self, n):
        out = []
        for k in range(n):
            self.f, self.rho, u, F = self.advance(self.f, self.rho, last=k == n - 1)
            self.u = u or self.u
            out.append(torch.stack([torch.as_tensor(v, dtype=torch.float64, device=self.f.device)
                                    for v in F]))
        return torch.stack(out)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("voxel", "place"):
        return None   # whole numbers
    cells = case["nx"] * case["ny"] * case["nz"]
    if cells * case["steps"] > (2e8 if kind in ("design", "adjoint") else 2.2e9):
        return None   # too long in plain float64
    lat = _Exact(case, seed)
    if kind == "channel":
        F = lat.steps(case["steps"])
        return dict(forces=F, ux=lat.u[0].flatten(), uy=lat.u[1].flatten(), uz=lat.u[2].flatten(),
                    rho=lat.rho.flatten())
    if kind == "frame":
        F = lat.steps(case["steps"])
        ux, uy, uz = (v.cpu().numpy() for v in lat.u)
        k = case["nz"] // 2
        view = np.sqrt(ux[k] ** 2 + uy[k] ** 2 + uz[k] ** 2) / case["u0"]
        view[lat.solid[k].cpu().numpy()] = np.nan
        p = _particles(case, seed)
        v = np.stack([_trilinear(a, p) for a in (ux, uy, uz)], 1)
        lim = np.array([case["nx"], case["ny"], case["nz"]]) - 1.5
        out = ((p < 0.5) | (p > lim)).any(1)
        v[out] = [case["u0"], 0.0, 0.0]
        return dict(forces=F, view=view, xyz=p + 2.0 * v, expired=None,
                    speed=np.sqrt((v * v).sum(1)) / case["u0"])
    box, s = _fraction(case, seed)
    st = torch.tensor(s.astype(np.float32).astype(np.float64) if kind == "design" else s,
                      device=lat.f.device, requires_grad=True)
    x0, y0, z0, x1, y1, z1 = box
    pad = (x0, case["nx"] - x1, y0, case["ny"] - y1, z0, case["nz"] - z1)

    def one(f, s_):
        g, _, _, F = lat.advance(f, lat.rho, torch.nn.functional.pad(s_, pad), last=False)
        return g, F[0]

    f, J = lat.f, 0.0
    for t in range(case["steps"]):
        f, fx = torch.utils.checkpoint.checkpoint(one, f, st, use_reentrant=False)
        if t >= case["steps"] - case["window"]:
            J = J + fx / case["window"]
    J.backward()
    return dict(J=J.detach(), grad=st.grad)


def _particles(case, seed):
    """The seeded smoke particles of a frame, spread over the tunnel."""
    r = np.random.default_rng(seed)
    return r.uniform(0.05, 0.95, (case["particles"], 3)) * [case["nx"], case["ny"], case["nz"]]


def _trilinear(a, p):
    q = p - 0.5
    i = np.clip(q.astype(np.int64), 0, np.array(a.shape[::-1]) - 2)
    t = q - i
    v = 0.0
    for c in range(8):
        o = np.array([c & 1, c >> 1 & 1, c >> 2])
        j = i + o
        v = v + np.prod(np.where(o, t, 1 - t), 1) * a[j[:, 2], j[:, 1], j[:, 0]]
    return v
