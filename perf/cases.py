"""The work that users of this framework have it do, as timed cases.

Three ways into the fluid step are covered, each over the range of sizes, storage types and boundary kinds
that the repository's own configurations, tests and benchmark use:

* one grid stepped by a program (``FluidGrid.step`` or ``step_coupled``), a control step at a time: the
  program hands in the solid's surface, steps the fluid ``steps`` times and reads the field (rho, u, pi) and
  the surface forces into device arrays;
* the same with the control step captured in a CUDA graph (``drive = "graph"``), as a latency-bound program
  does it;
* the serving pool (``serving.Pool``): actions in, one control step of 10 substeps for every admitted
  episode, output records back on the host.

``exact`` restates the step in 64-bit torch arithmetic from the lattice-Boltzmann equations; it uses none of
the kernels.  Link membership is decided there in 64 bits as well, so a link that passes within rounding of
an element's edge can differ from the 32-bit geometry of the step.
"""
import ctypes
import itertools
import math
import random

import numpy as np
import torch

from freeflow_b200 import DeviceSurface, FluidGrid, _capi, serving, workloads
from freeflow_b200.grid import VolumeSurface

DEVICE = "cuda"
STORED = {"f32": 4, "f16": 2, "bf16": 2}
MOMENTS = {2: 6, 3: 10}
# floating-point operations of one cell update (reconstruction, streaming clamp, raw moments, collision)
FLOPS = {2: 120, 3: 400}
TAIL = 0.05           # lattice speed of a swimmer's tail
SUBSTEPS = 10         # fluid steps per control step of the pool
POOL_SIZES = serving.SERVING_SIZES


def _grid(name, dim, nx, ny, nz, storage, scene, drive, steps):
    return dict(name=name, kind="grid", dim=dim, nx=nx, ny=ny, nz=nz, storage=storage, scene=scene, drive=drive,
                steps=steps)


def _pool(name, episodes, storage, mix, observe):
    return dict(name=name, kind="pool", episodes=episodes, storage=storage, mix=mix, observe=observe)


def listed():
    return [
        # fixed cylinder in a channel: a launch-bound 2D program, the surface never moves
        _grid("cylinder-256x128-f32", 2, 256, 128, 1, "f32", "cylinder", "loop", 10),
        # the reference's 2D fish scene: open on four sides, surface handed in before every step
        _grid("fish-1200x400-f32", 2, 1200, 400, 1, "f32", "open", "loop", 10),
        # the same in reduced storage with the control step captured in a graph
        _grid("fish-1200x400-f16", 2, 1200, 400, 1, "f16", "open", "graph", 10),
        # odd sizes, closed tank, forces scattered to a volume mesh (a deformable solver's step)
        _grid("tank-509x187-bf16", 2, 509, 187, 1, "bf16", "tank", "coupled", 10),
        # the smallest 3D scene: latency and launches
        _grid("channel-64x32x32-f32", 3, 64, 32, 32, "f32", "channel", "graph", 10),
        # periodic Taylor-Green-sized box without a solid
        _grid("vortex-128-f32", 3, 128, 128, 128, "f32", "vortex", "loop", 10),
        # ragged 3D channel, coupled to a volume mesh, reduced storage
        _grid("channel-189x93x101-bf16", 3, 189, 93, 101, "bf16", "channel", "coupled", 10),
        # the 3D swimmer channel in both storages of the benchmark
        _grid("channel-384x192x192-f32", 3, 384, 192, 192, "f32", "channel", "loop", 10),
        _grid("channel-384x192x192-f16", 3, 384, 192, 192, "f16", "channel", "loop", 10),
        # a few environments whose flow field is part of the observation
        _pool("pool-4-observed-f16", 4, "f16", 1, True),
        # serving mixes at two of the benchmark's concurrencies
        _pool("pool-64-f16", 64, "f16", 2, False),
        _pool("pool-256-f16", 256, "f16", 3, False),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    what = rng.random()
    storage = rng.choice(["f32", "f16", "bf16"])
    if what < 0.3:
        nx = _log(rng, 160, 1400)
        c = _grid(None, 2, nx, _log(rng, 96, max(97, min(480, nx))), 1, storage,
                  rng.choice(["cylinder", "open", "tank"]), rng.choice(["loop", "graph", "coupled"]),
                  2 * rng.randint(1, 5))
    elif what < 0.75:
        ny = _log(rng, 28, 190)
        nx = max(40, min(380, int(ny * rng.uniform(1.0, 2.2))))
        nz = max(24, min(190, int(ny * rng.uniform(0.7, 1.2))))
        c = _grid(None, 3, nx, ny, nz, storage, rng.choice(["channel", "channel", "vortex"]),
                  rng.choice(["loop", "graph", "coupled"]), 2 * rng.randint(1, 4))
        if c["scene"] == "vortex" and c["drive"] == "coupled":
            c["drive"] = "loop"
    else:
        n = _log(rng, 1, 200)
        c = _pool(None, n, rng.choice(["f16", "f16", "f32", "bf16"]), rng.randint(10, 9999), n <= 4)
    del c["name"]
    return c


# ------------------------------------------------------------------------------------------------- scenes
def _scene(case, seed):
    """Grid arguments, flags, initial moments (SoA, on the GPU) and the surface's table of positions and
    velocities over one period (a multiple of 10 steps), everything from the seed."""
    rng = np.random.default_rng(seed)
    dim, nx, ny, nz = case["dim"], case["nx"], case["ny"], case["nz"]
    scene, u_in, periodic = case["scene"], 0.05, 0
    dx, dt = (0.005, 0.0025) if dim == 2 else (0.01, 0.005)
    nu, density = {"cylinder": (0.016, 1000.0), "open": (0.01, 10.0), "tank": (0.01, 10.0), "vortex": (0.005, 1.0),
                   "channel": (0.01, 500.0)}[scene]
    bc = [0.0] * 6
    if scene == "cylinder":
        flags = workloads.channel_flags_2d(nx, ny)
        bc[0] = u_in
    elif scene in ("open", "tank"):
        sides = ([workloads.OUTLET_DOWN, workloads.OUTLET_UP, workloads.OUTLET_LEFT, workloads.OUTLET_RIGHT]
                 if scene == "open" else [workloads.WALL] * 4)
        f = np.full((ny, nx), workloads.FLUID, np.uint8)
        f[0, :], f[-1, :], f[:, 0], f[:, -1] = sides
        flags = f.reshape(-1)
    elif scene == "channel":
        flags = workloads.channel_flags_3d(nx, ny, nz)
        bc[0] = u_in
    else:
        flags, periodic = np.full(nx * ny * nz, workloads.FLUID, np.uint8), 7
    grid = dict(dim=dim, nx=nx, ny=ny, nz=nz, fluid_viscosity=nu, fluid_density=density, fluid_dx=dx, dt=dt,
                boundary_velocities=bc, storage=case["storage"], periodic=periodic)
    moments = _flow(rng, dim, nx, ny, nz, flags, bc[0])
    return grid, flags, moments, _surface(case, rng, dx, dt)


def _flow(rng, dim, nx, ny, nz, flags, u_in):
    """A developed-looking state: a few Fourier modes of velocity (0.03) and density (1e-3), equilibrium
    stress plus a small non-equilibrium part; boundary nodes at rest, inlets at the inlet velocity."""
    shape = (nz, ny, nx)
    axes = [torch.arange(n, device=DEVICE, dtype=torch.float64) * (2.0 * math.pi / n) for n in shape]

    def waves(amplitude, modes=3):
        out = torch.zeros(shape, device=DEVICE, dtype=torch.float32)
        for _ in range(modes):
            k, ph = rng.integers(1, 5, 3), rng.uniform(0.0, 2.0 * math.pi, 3)
            w = [torch.sin(int(k[a]) * axes[a] + ph[a]).float() if shape[a] > 1 else torch.ones(1, device=DEVICE)
                 for a in range(3)]
            out += (amplitude * float(rng.uniform(0.3, 1.0)) / modes) * (w[0][:, None, None] * w[1][:, None] * w[2])
        return out.reshape(-1)

    m = torch.empty((MOMENTS[dim], nx * ny * nz), device=DEVICE, dtype=torch.float32)
    t = torch.as_tensor(flags, device=DEVICE)
    fluid, inlet = t == workloads.FLUID, t == workloads.INLET_LEFT
    m[0] = torch.where(fluid, 1.0 + waves(1e-3), 1.0)
    for a in range(dim):
        base = 0.6 * u_in if a == 0 else 0.0
        m[1 + a] = torch.where(fluid, base + waves(0.03), 0.0)
    m[1] = torch.where(inlet, u_in, m[1])
    for k, (a, b) in enumerate(_pairs(dim)):
        m[1 + dim + k] = m[1 + a] * m[1 + b] + torch.where(fluid, waves(2e-4), 0.0)
    return m


def _pairs(dim):
    return [(0, 0), (1, 1), (0, 1)] if dim == 2 else [(0, 0), (1, 1), (2, 2), (0, 1), (1, 2), (0, 2)]


def _surface(case, rng, dx, dt):
    """(elements, positions, velocities) with positions and velocities (T, nv, dim) on the GPU, or None."""
    dim, nx, ny, nz, scene = case["dim"], case["nx"], case["ny"], case["nz"], case["scene"]
    if scene == "vortex":
        return None
    if scene == "cylinder":
        r = 0.125 * ny
        v, e = workloads.circle_polygon(0.25 * nx + rng.uniform(-0.4, 0.4), 0.5 * ny + rng.uniform(-0.4, 0.4), r,
                                        max(24, int(8 * r) // 2 * 2))
        pos = torch.as_tensor((v * dx).astype(np.float32), device=DEVICE)[None]
        return e, pos, torch.zeros_like(pos)
    if dim == 2:
        length = 0.4 * ny
        p, e = workloads.fish_outline(length, 99, rng=rng, jitter=1e-3)
        centre = np.array([0.25 * nx, 0.5 * ny])
        s = np.clip(p[:, 0] / length, 0.0, 1.0)
        x, amp, axis = p[:, 0], workloads.carangiform_envelope(s, length), 1
    else:
        length = 0.3 * nx
        n = max(8, min(64, int(length * 0.6)))
        p, e = workloads.ellipsoid_mesh(0.5 * length, 0.05 * max(ny, 40), 0.05 * max(nz, 40), n, n)
        p = p + rng.uniform(-1e-3, 1e-3, p.shape)
        centre = np.array([0.35 * nx, 0.5 * ny, 0.5 * nz]) + rng.uniform(-0.3, 0.3, 3)
        x, axis = p[:, 0] + 0.5 * length, 2
        s = np.clip(x / length, 0.0, 1.0)
        amp = 0.08 * length * s * s
    # one period of the body wave, long enough that the tail moves at TAIL cells per step
    period = max(20, int(2.0 * math.pi * float(np.abs(amp).max()) / TAIL) // 10 * 10)
    om = 2.0 * math.pi / period
    ph = torch.as_tensor(2.0 * math.pi / length * x, device=DEVICE)[None] - om * torch.arange(
        period, device=DEVICE, dtype=torch.float64)[:, None]
    a = torch.as_tensor(amp, device=DEVICE)
    pos = torch.as_tensor((centre + p) * dx, device=DEVICE).repeat(period, 1, 1)
    vel = torch.zeros_like(pos)
    pos[:, :, axis] += a * torch.sin(ph) * dx
    vel[:, :, axis] = -a * om * torch.cos(ph) * (dx / dt)
    return e, pos.float().contiguous(), vel.float().contiguous()


def _mix(case, seed):
    """The pool's episodes (their sizes from the case, everything else from the seed) and 64 control steps of
    actions."""
    sizes = random.Random(case["mix"])
    rng = np.random.default_rng(seed)
    specs = []
    for _ in range(case["episodes"]):
        nx, ny = sizes.choice(POOL_SIZES)
        specs.append(serving.make_episode(nx, ny, seed=int(rng.integers(0, 2 ** 31)), length=1000,
                                          sides="walls" if sizes.random() < 0.25 else "outlets"))
    return specs, rng.uniform(-1.0, 1.0, (64, case["episodes"], 8)).astype(np.float32)


# ---------------------------------------------------------------------------------------------- the program
def prepare(case, seed):
    if case["kind"] == "pool":
        specs, actions = _mix(case, seed)
        scratch = serving.Pool(storage=case["storage"], budget_bytes=1 << 20, max_episodes=1)
        need = sum(scratch.episode_bytes(s) for s in specs)
        scratch.close()
        pool = serving.Pool(storage=case["storage"], budget_bytes=need + (1 << 20), max_episodes=case["episodes"],
                            substeps=SUBSTEPS)
        return dict(case=case, pool=pool, slots=[pool.admit(s) for s in specs], actions=actions, turn=0)
    grid_args, flags, moments, table = _scene(case, seed)
    g = FluidGrid(**grid_args)
    g.set_flags(flags)
    _set_field(g, moments)
    st = dict(case=case, grid=g, field=torch.empty_like(moments), table=table, turn=0, surface=None)
    if table is not None:
        e, pos, vel = table
        p0, v0 = pos[0].cpu().numpy(), vel[0].cpu().numpy()
        if case["drive"] == "coupled":
            vol, where = _volume_map(len(p0), seed)
            vp = np.zeros((vol, case["dim"]), np.float32)
            vv = np.zeros_like(vp)
            vp[where], vv[where] = p0, v0
            st["surface"] = VolumeSurface(vp, vv, where, e)
            st["where"] = torch.as_tensor(where.astype(np.int64), device=DEVICE)
        else:
            st["surface"] = DeviceSurface(p0, v0, e)
    if case["drive"] == "graph":
        _capture(st, moments)
    return st


def _volume_map(nv, seed):
    vol = nv + nv // 2
    return vol, np.random.default_rng(seed + 1).permutation(vol)[:nv].astype(np.uint32)


def _set_field(g, moments):
    """The C ABI's device-to-device form of FluidGrid.set_moments."""
    _capi.check(_capi.load().ffs_lbm_set_moments(g.handle, ctypes.c_void_p(moments.data_ptr()), _capi.LAYOUT_SOA,
                                                 _capi.MEM_DEVICE, _capi.BUF_BOTH, None), "set_moments")


def _get_field(g, out, stream=None):
    """The C ABI's device-to-device form of FluidGrid.get_moments."""
    _capi.check(_capi.load().ffs_lbm_get_moments(g.handle, ctypes.c_void_p(out.data_ptr()), _capi.LAYOUT_SOA,
                                                 _capi.MEM_DEVICE, _capi.BUF_CURRENT,
                                                 ctypes.c_void_p(stream.cuda_stream) if stream else None),
                "get_moments")


def _capture(st, moments):
    """Captures one control step: surface hand-over and fluid steps, then the field's read-out.  The first
    eager step sets the grid up; the field is put back afterwards."""
    case, g, surf = st["case"], st["grid"], st["surface"]
    g.step(surf)
    torch.cuda.synchronize()
    _set_field(g, moments)
    moving = surf is not None and st["table"][1].shape[0] > 1
    if moving:
        st["pos"] = st["table"][1][:case["steps"]].clone()
        st["vel"] = st["table"][2][:case["steps"]].clone()
    torch.cuda.synchronize()
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        if surf is not None:
            surf.forces.zero_()
        for j in range(case["steps"]):
            if moving:
                surf.vertices.copy_(st["pos"][j])
                surf.velocities.copy_(st["vel"][j])
            g.step(surf, stream=stream)
        _get_field(g, st["field"], stream)
    st["graph"] = graph


def _window(st):
    """Rows of the surface table that this pass's steps take."""
    n, period = st["case"]["steps"], st["table"][1].shape[0]
    at = [(st["turn"] * n + j) % period for j in range(n)]
    st["turn"] += 1
    return at


def run(st):
    case = st["case"]
    if case["kind"] == "pool":
        return _run_pool(st)
    g, surf, dim = st["grid"], st["surface"], case["dim"]
    if case["drive"] == "graph":
        if "pos" in st:
            at = _window(st)
            if at[-1] == at[0] + len(at) - 1:
                st["pos"].copy_(st["table"][1][at[0]:at[0] + len(at)])
                st["vel"].copy_(st["table"][2][at[0]:at[0] + len(at)])
            else:
                st["pos"].copy_(st["table"][1][at])
                st["vel"].copy_(st["table"][2][at])
        st["graph"].replay()
    elif surf is None:
        for _ in range(case["steps"]):
            g.step()
        _get_field(g, st["field"])
    else:
        _, pos, vel = st["table"]
        at = _window(st)
        if case["drive"] == "loop":
            surf.forces.zero_()
        for k in at:
            if case["drive"] == "coupled":
                if pos.shape[0] > 1:
                    # the solid solver's new state, written where its mesh lives
                    surf.volume_positions.index_copy_(0, st["where"], pos[k])
                    surf.volume_velocities.index_copy_(0, st["where"], vel[k])
                g.step_coupled(surf)
            else:
                if pos.shape[0] > 1:
                    surf.update(pos[k], vel[k])
                g.step(surf)
        _get_field(g, st["field"])
    f = st["field"]
    out = {"rho": f[0], "velocity": f[1:1 + dim], "stress": f[1 + dim:]}
    if surf is not None:
        out["forces"] = surf.volume_forces if case["drive"] == "coupled" else surf.forces
    return out


def _run_pool(st):
    pool, slots = st["pool"], st["slots"]
    pool.set_actions(slots, st["actions"][st["turn"] % 64])
    st["turn"] += 1
    pool.advance()
    rec = pool.collect_many(slots)
    out = {"energy": rec["energy"].copy(), "force": rec["force"].copy(), "torque": rec["torque"].copy(),
           "status": rec["status"].astype(np.int64)}
    if st["case"]["observe"]:
        out["vertex_forces"] = [pool.collect(s, forces=True)[1] for s in slots]
        fields = [pool.get_moments(s) for s in slots]
        out["rho"] = [m[:, 0] for m in fields]
        out["velocity"] = [m[:, 1:3] for m in fields]
        out["stress"] = [m[:, 3:] for m in fields]
    return out


# ------------------------------------------------------------------------------------------------ accounting
def work(case):
    if case["kind"] == "pool":
        sizes = random.Random(case["mix"])
        cells = 0
        for _ in range(case["episodes"]):
            nx, ny = sizes.choice(POOL_SIZES)
            sizes.random()
            cells += nx * ny
        s = STORED[case["storage"]]
        read_out = cells * 6 * (s + 4) if case["observe"] else 0
        return {"bytes": SUBSTEPS * cells * (12 * s + 1) + read_out, "flops": SUBSTEPS * cells * FLOPS[2]}
    dim, s = case["dim"], STORED[case["storage"]]
    cells, nm = case["nx"] * case["ny"] * case["nz"], MOMENTS[dim]
    return {"bytes": case["steps"] * cells * (2 * nm * s + 1) + cells * nm * (s + 4),
            "flops": case["steps"] * cells * FLOPS[dim]}


def tolerance(case):
    # The stress decides: it is 1e-4 to 1e-3 of the density's scale, so what is a few units in the last place of
    # the raw moments is most there.  Measured against exact(): 32-bit storage, stress 2.8e-4 (velocity 6e-6);
    # 16-bit storage, stress 1e-2 (velocity 6e-4), pools 2.6e-3.  In 16-bit storage the stored velocity is rounded
    # stochastically with a dither taken from the density's bits, so any other rounding of the density gives
    # another dither, and two correct implementations differ by about as much as each is off.
    if case["storage"] == "f32":
        return {"rel": 1.2e-3, "max": 2e-2}
    return {"rel": 1e-2 if case["kind"] == "pool" else 3e-2, "max": 0.6}


# ------------------------------------------------------------------------------------- the step in 64 bits
FLUID, SOLID_DYNAMIC = 1, 4
BOUNCE = {2: (3, 5, 6, 7, 10, 11), 3: (3, 5, 6, 7, 8, 9, 10, 11)}
# outlet node type -> (axis, outward sign); axes x, y, z = 0, 1, 2
OUTLETS = {2: {19: (0, -1), 20: (0, 1), 21: (1, 1), 22: (1, -1)},
           3: {19: (0, -1), 20: (0, 1), 21: (2, 1), 22: (2, -1), 23: (1, -1), 24: (1, 1)}}


class _Exact:
    """The moment-encoded step of one grid in 64-bit torch arithmetic, arrays as (nz, ny, nx)."""

    def __init__(self, dim, nx, ny, nz, flags, moments, viscosity, density, dx, dt, periodic):
        self.dim, self.shape, self.periodic = dim, (nz, ny, nx), periodic
        self.m = [moments.double().reshape(-1, nz, ny, nx) for _ in range(2)]
        self.m[1] = self.m[0].clone()
        self.type = torch.as_tensor(np.asarray(flags).reshape(nz, ny, nx).astype(np.int64), device=DEVICE)
        self.omega = 1.0 / (3.0 * float(np.float32(viscosity)) + 0.5)
        mass = np.float32(density * dx ** dim)
        self.cf = float(np.float32(float(mass) * dx / (dt * dt)))
        self.cl, self.ct = float(np.float32(dx)), float(np.float32(dt))
        self.c = [c for c in itertools.product((0, 1, -1), repeat=dim)]
        self.bounce = sum((self.type == b) for b in BOUNCE[dim]) > 0
        self.updated = (self.type == FLUID) | (self.type == SOLID_DYNAMIC)

    def _shifted(self, f, c, wrap):
        """f at x - c for every x: wrapped, or with the pull's halo (wraps low, stays high) on open axes."""
        for a in range(self.dim):
            if c[a] == 0:
                continue
            ax = 2 - a
            n = self.shape[ax]
            i = torch.arange(n, device=DEVICE) - c[a]
            if wrap or self.periodic >> a & 1:
                i = i % n
            else:
                i = torch.where((i < 0) | (i >= n), n - 1, i)
            f = f.index_select(ax, i)
        return f

    def _coefficients(self, m):
        d, r = self.dim, m[0]
        u, p = m[1:1 + d], {k: m[1 + d + i] for i, k in enumerate(_pairs(d))}
        q = {}
        for a in range(d):
            for b in range(d):
                if a != b:
                    ab = p[(min(a, b), max(a, b))]
                    if d == 2:    # the 2D expansion carries no density on the stress terms of its third order
                        q[(a, b)] = 9.0 * (p[(a, a)] * u[b] + 2.0 * u[a] * (ab - r * u[a] * u[b]))
                    else:
                        q[(a, b)] = 9.0 * r * (p[(a, a)] * u[b] + 2.0 * u[a] * (ab - u[a] * u[b]))
        xyz = None
        if d == 3:
            xyz = 27.0 * r * (p[(0, 1)] * u[2] + p[(1, 2)] * u[0] + p[(0, 2)] * u[1] - 2.0 * u[0] * u[1] * u[2])
        return r, u, p, q, xyz

    def _population(self, co, c):
        r, u, p, q, xyz = co
        d = self.dim
        g = [1.0 if x else -0.5 for x in c]
        f = r.clone()
        for a in range(d):
            f = f + 3.0 * r * (u[a] * c[a] + p[(a, a)] * g[a])
            for b in range(d):
                if a < b and c[a] * c[b]:
                    f = f + (9.0 * c[a] * c[b]) * (r * p[(a, b)])
                if a != b and c[b]:
                    f = f + (g[a] * c[b]) * q[(a, b)]
        if d == 3 and c[0] * c[1] * c[2]:
            f = f + (c[0] * c[1] * c[2]) * xyz
        return f * math.prod(1.0 / 6.0 if x else 2.0 / 3.0 for x in c)

    def step(self, surface=None):
        """One step; surface = (elements, positions, velocities).  Returns the vertex forces, or None."""
        d, src, dst = self.dim, self.m[0], self.m[1]
        co = self._coefficients(src)
        pops = {c: self._population(co, c) for c in self.c}
        pulled = {}
        for c in self.c:
            f = self._shifted(pops[c], c, False)
            if any(c):
                f = torch.where(self._shifted(self.bounce, c, True), pops[tuple(-x for x in c)], f)
            pulled[c] = f.clamp_min(0.0)
        forces = self._links(surface, src, pops, pulled) if surface is not None else None
        del pops
        raw = [sum(pulled[c] for c in self.c)]
        raw += [sum(c[a] * pulled[c] for c in self.c if c[a]) for a in range(d)]
        raw += [sum(c[a] * c[b] * pulled[c] for c in self.c if c[a] * c[b]) for a, b in _pairs(d)]
        rho, w = raw[0], self.omega
        u = [raw[1 + a] / rho for a in range(d)]
        u2, tr = sum(x * x for x in u) / d, sum(raw[1 + d + a] for a in range(d)) / d
        new = [rho] + u
        for i, (a, b) in enumerate(_pairs(d)):
            if a == b:
                new.append((1.0 - w) * (raw[1 + d + i] - tr) / rho + u2 + w * (u[a] * u[a] - u2))
            else:
                new.append((1.0 - w) * raw[1 + d + i] / rho + w * u[a] * u[b])
        for k in range(len(new)):
            dst[k] = torch.where(self.updated, new[k], dst[k])
        for t, (a, s) in OUTLETS[d].items():
            at = self.type == t
            if not bool(at.any()):
                continue
            n = tuple(s if k == a else 0 for k in range(d))
            at &= self._shifted(self.type, n, True) == FLUID
            up = self._shifted(dst[1 + a], n, True)
            dst[1 + a] = torch.where(at & (s * up > 0), up, dst[1 + a])
            k = 1 + d + _pairs(d).index((a, a))
            dst[k] = torch.where(at, up * up, dst[k])
        self.m = [dst, src]
        return forces

    def _hits(self, e, pos, cells, c):
        """(hit, depth, weights of the element's vertices) of the links cells -> cells - c."""
        p1 = cells * self.cl
        step = torch.tensor([-x * self.cl for x in c], device=DEVICE, dtype=torch.float64)
        v = pos[e][:, None]                         # (ne, 1, vertex, axis)
        if self.dim == 2:
            a, b = v[..., 0, :], v[..., 1, :]
            n = torch.stack([a[..., 1] - b[..., 1], b[..., 0] - a[..., 0]], -1)
            den = -(step * n).sum(-1)
            t1 = ((b - p1 - step) * n).sum(-1) / den
            at = p1 + (1.0 - t1)[..., None] * step
            hit = (t1 > 0) & (t1 < 1) & ((a[..., 0] - at[..., 0]) * (b[..., 0] - at[..., 0]) < 0)
            w0 = (b - at).norm(dim=-1) / (b - a).norm(dim=-1)
            return hit & torch.isfinite(t1), 1.0 - t1, torch.stack([w0, 1.0 - w0], -1)
        v0 = v[..., 0, :]
        e1, e2 = v[..., 1, :] - v0, v[..., 2, :] - v0
        n = torch.linalg.cross(e1, e2)
        n = n / n.norm(dim=-1, keepdim=True)
        ns = (n * step).sum(-1)
        t = (n * (v0 - p1)).sum(-1) / ns
        w = p1 + t[..., None] * step - v0
        d00, d01, d11 = (e1 * e1).sum(-1), (e1 * e2).sum(-1), (e2 * e2).sum(-1)
        d20, d21 = (w * e1).sum(-1), (w * e2).sum(-1)
        den = d00 * d11 - d01 * d01
        b1, b2 = (d11 * d20 - d01 * d21) / den, (d00 * d21 - d01 * d20) / den
        hit = (ns.abs() > 1e-6 * step.norm()) & (t >= 0) & (t <= 1) & (b1 >= -1e-6) & (b2 >= -1e-6) & (b1 + b2 <= 1 + 1e-6)
        return hit, t, torch.stack([1.0 - b1 - b2, b1, b2], -1)

    def _links(self, surface, src, pops, pulled):
        d = self.dim
        e = torch.as_tensor(np.asarray(surface[0]).astype(np.int64), device=DEVICE)
        pos, vel = surface[1].double(), surface[2].double()
        size = torch.tensor(self.shape[::-1][:d], device=DEVICE)
        lo = torch.floor(pos[e].amin(1) / self.cl).long() - 1
        ext = (torch.floor(pos[e].amax(1) / self.cl).long() + 2 - lo).amax(0).tolist()
        off = torch.cartesian_prod(*[torch.arange(k, device=DEVICE) for k in ext])
        cells = lo[:, None] + off                                   # (ne, box, axis)
        ok = ((cells >= 0) & (cells < size)).all(-1)
        stride = torch.tensor([1, self.shape[2], self.shape[1] * self.shape[2]][:d], device=DEVICE)
        flat = (cells * stride).sum(-1)
        forces = torch.zeros_like(pos)
        for c in self.c:
            if not any(c):
                continue
            hit, depth, bary = self._hits(e, pos, cells.double(), c)
            back = cells - torch.tensor(c, device=DEVICE)
            hit &= ok & ((back >= 0) & (back < size)).all(-1)
            el, bx = hit.nonzero(as_tuple=True)
            cell = flat[el, bx]
            keep = self.updated.reshape(-1)[cell] & ~self._shifted(self.bounce, c, True).reshape(-1)[cell]
            el, bx, cell = el[keep], bx[keep], cell[keep]
            if not len(el):
                continue
            # the nearest element owns the link: depth in 1/32768 of it, then the element's number
            order = (((cell << 16) + (depth[el, bx] * 32768.0).long()) << 18) + el
            order, perm = order.sort()
            first = torch.ones_like(order, dtype=torch.bool)
            first[1:] = (order[1:] >> 34) != (order[:-1] >> 34)
            perm = perm[first]
            el, bx, cell = el[perm], bx[perm], cell[perm]
            w = bary[el, bx]
            uw = (vel[e[el]] * w[..., None]).sum(1) * (self.ct / self.cl)
            mc = src.reshape(src.shape[0], -1)[:, cell]
            mw = [mc[0]] + [uw[:, a] for a in range(d)]
            mw += [mc[1 + d + i] + uw[:, a] * uw[:, b] - mc[1 + a] * mc[1 + b] for i, (a, b) in enumerate(_pairs(d))]
            fout = self._population(self._coefficients(torch.stack(mw)), c)
            fin = pops[tuple(-x for x in c)].reshape(-1)[cell].clamp_min(0.0)
            pulled[c].reshape(-1)[cell] = fout
            cv = torch.tensor(c, device=DEVICE, dtype=torch.float64)
            F = fin[:, None] * (-cv - uw) - fout[:, None] * (cv - uw)
            for j in range(d):
                forces.index_add_(0, e[el, j], F * w[:, j, None])
        return forces * self.cf


def exact(case, seed):
    if case["kind"] == "pool":
        return _exact_pool(case, seed)
    g, flags, moments, table = _scene(case, seed)
    d = case["dim"]
    x = _Exact(d, case["nx"], case["ny"], case["nz"], flags, moments, g["fluid_viscosity"], g["fluid_density"],
               g["fluid_dx"], g["dt"], g["periodic"])
    total = None
    for k in range(case["steps"]):
        s = None if table is None else (table[0], table[1][k % len(table[1])], table[2][k % len(table[2])])
        f = x.step(s)
        if f is not None:
            total = f if total is None or case["drive"] == "coupled" else total + f
    m = x.m[0].reshape(MOMENTS[d], -1)
    out = {"rho": m[0], "velocity": m[1:1 + d], "stress": m[1 + d:]}
    if total is not None:
        if case["drive"] == "coupled":
            vol, where = _volume_map(len(total), seed)
            out["forces"] = torch.zeros((vol, d), device=DEVICE, dtype=torch.float64)
            out["forces"][torch.as_tensor(where.astype(np.int64), device=DEVICE)] = total
        else:
            out["forces"] = total
    return out


def _exact_pool(case, seed):
    if case["episodes"] > 64:
        return None
    specs, actions = _mix(case, seed)
    out = {k: [] for k in ("energy", "force", "torque", "vertex_forces", "rho", "velocity", "stress")}
    for i, sp in enumerate(specs):
        rest = torch.as_tensor(sp.rest, device=DEVICE).double()
        m = torch.zeros((6, sp.ncell), device=DEVICE, dtype=torch.float64)
        m[0] = 1.0
        x = _Exact(2, sp.nx, sp.ny, 1, sp.flags, m, sp.viscosity, sp.density, sp.dx, sp.dt, 0)
        seg = torch.as_tensor(sp.segment.astype(np.int64), device=DEVICE)
        act = torch.as_tensor(actions[0, i], device=DEVICE).double()
        amp = torch.as_tensor(sp.amplitude, device=DEVICE).double() * (1.0 + 0.5 * torch.where(seg >= 0, act[seg], 0.0))
        sk, ck = (torch.as_tensor(a, device=DEVICE).double() for a in (sp.sin_kx, sp.cos_kx))
        centre = rest.mean(0)
        energy, force, torque = 0.0, torch.zeros(2, device=DEVICE, dtype=torch.float64), 0.0
        for j in range(SUBSTEPS):
            th = sp.omega * (sp.t0 + j * sp.dt)
            pos, vel = rest.clone(), torch.zeros_like(rest)
            pos[:, 1] += amp * (sk * math.cos(th) - ck * math.sin(th))
            vel[:, 1] = -amp * sp.omega * (ck * math.cos(th) + sk * math.sin(th))
            f = x.step((sp.elements, pos.float(), vel.float()))
            energy = energy + torch.clamp_min(-(f * vel).sum(), 0.0) * sp.dt
            force = force + f.sum(0) / SUBSTEPS
            r = pos - centre
            torque = torque + (r[:, 0] * f[:, 1] - r[:, 1] * f[:, 0]).sum() / SUBSTEPS
        out["energy"].append(energy)
        out["force"].append(force)
        out["torque"].append(torque)
        out["vertex_forces"].append(f)
        out["rho"].append(x.m[0][0].reshape(-1))
        out["velocity"].append(x.m[0][1:3].reshape(2, -1).T.contiguous())
        out["stress"].append(x.m[0][3:].reshape(3, -1).T.contiguous())
    res = {"energy": torch.stack(out["energy"]), "force": torch.stack(out["force"]),
           "torque": torch.stack(out["torque"]), "status": None}
    if case["observe"]:
        for k in ("vertex_forces", "rho", "velocity", "stress"):
            res[k] = out[k]
    return res
