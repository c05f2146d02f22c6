"""Bodies that reach the cells next to an outlet: such a cell has links and
feeds an outlet node, which keeps its old normal velocity when the new one
points inward.  The node must get the link cell's final value and nothing of
the plain update that the dense pass may have made first, in every order of
link detection and dense pass:

  * the step as it runs (detection beside the dense pass) and with detection
    first (serial stage timing): the same bits, step after step
  * against the ref32 oracle in FP32: moments max |diff| <= 4e-6 (the bound of
    test_gpu_random_flags.py)
  * the serving pool and one grid per episode: the same bits, also where the
    first control step times the pool's work units

The walls move inward and outward by turns while the fluid goes outward, so that
the plain and the final normal velocity differ in sign in many of these cells.
"""
import numpy as np
import pytest

from freeflow_b200 import serving as S
from freeflow_b200 import workloads as W

from helpers import make_gpu, make_oracle, max_abs

pytestmark = pytest.mark.gpu


def _scene2(nx, ny):
    """Outlets on four sides, flow out at the right and the top; a circle across either face."""
    wl = W.cylinder_channel_2d(nx=max(nx, 64), ny=max(ny, 48), seed=1)
    wl.nx, wl.ny = nx, ny
    rng = np.random.default_rng(3)
    u = np.array([0.03, 0.02]) + rng.uniform(-5e-3, 5e-3, (nx * ny, 2))
    wl.moments = W.equilibrium_moments(1.0 + rng.uniform(-1e-3, 1e-3, nx * ny), u)
    f = np.full((ny, nx), W.FLUID, np.uint8)
    f[0, :], f[-1, :], f[:, 0], f[:, -1] = W.OUTLET_DOWN, W.OUTLET_UP, W.OUTLET_LEFT, W.OUTLET_RIGHT
    wl.flags = f.reshape(-1)
    a, e = W.circle_polygon(nx - 6.3, 0.45 * ny, 7.2, 40)
    b, e2 = W.circle_polygon(0.4 * nx, ny - 5.4, 6.1, 36)
    wl.elements = np.concatenate([e, e2 + len(a)]).astype(np.uint32)
    return wl, np.concatenate([a, b])


def _scene3(nx, ny, nz):
    """The 3D channel with an ellipsoid across its outlet face."""
    wl = W.swimmer_3d(nx=nx, ny=ny, nz=nz, nlat=10, nlon=14, seed=2)
    rng = np.random.default_rng(4)
    n = nx * ny * nz
    u = np.array([0.03, 0.0, 0.0]) + rng.uniform(-5e-3, 5e-3, (n, 3))
    wl.moments = W.equilibrium_moments(1.0 + rng.uniform(-1e-3, 1e-3, n), u)
    p, e = W.ellipsoid_mesh(6.0, 5.0, 5.5, 10, 14)
    wl.elements = e
    return wl, p + np.array([nx - 5.6, 0.5 * ny, 0.5 * nz])


def _surface(wl, rest, step):
    """Vertices in place, a velocity that turns every third step (0.06 cells a step)."""
    scale = wl.fluid_dx / wl.dt
    u = np.zeros_like(rest)
    u[:, 0] = (-0.06 if step // 3 % 2 == 0 else 0.05) * scale
    u[:, 1] = (-0.06 if step % 2 == 0 else 0.04) * scale
    return (rest * wl.fluid_dx).astype(np.float32), u.astype(np.float32)


def _states(wl, rest, storage, serial, steps, ref_half=False):
    from freeflow_b200 import DeviceSurface

    els, wl.elements = wl.elements, None
    g, _ = make_gpu(wl, storage, ref_half)
    wl.elements = els
    if serial:
        g.profile(True, serial=True)
    s = DeviceSurface(*_surface(wl, rest, 0), els, with_forces64=True)
    out = []
    for k in range(steps):
        s.update(*_surface(wl, rest, k))
        g.step(s)
        out.append(g.get_moments())
    status = g.status()
    forces = s.forces64.cpu().numpy().copy()
    g.close()
    return out, forces, status


SCENES = [(_scene2, (64, 48)), (_scene2, (131, 75)), (_scene2, (700, 520)), (_scene3, (40, 28, 30)), (_scene3, (67, 33, 29))]


@pytest.mark.parametrize("storage", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("scene,size", SCENES, ids=["x".join(map(str, s[1])) for s in SCENES])
def test_detection_first_or_beside(cuda, scene, size, storage):
    wl, rest = scene(*size)
    first, f0, st0 = _states(wl, rest, storage, True, 9)
    assert st0 == 0 and np.abs(f0).max() > 0
    for _ in range(3):
        beside, f1, st1 = _states(wl, rest, storage, False, 9)
        assert st1 == 0
        for k, (a, b) in enumerate(zip(first, beside)):
            assert np.array_equal(a, b), f"step {k}: {int((a != b).any(axis=1).sum())} cells differ"
        assert np.array_equal(f0, f1)


@pytest.mark.parametrize("scene,size", SCENES, ids=["x".join(map(str, s[1])) for s in SCENES])
def test_against_oracle(cuda, scene, size):
    wl, rest = scene(*size)
    got, _, _ = _states(wl, rest, "f32", False, 6)
    o = make_oracle(wl)
    outlets = np.isin(wl.flags, [W.OUTLET_DOWN, W.OUTLET_UP, W.OUTLET_LEFT, W.OUTLET_RIGHT])
    assert outlets.sum() > 0
    for k in range(6):
        v, u = _surface(wl, rest, k)
        o.step(v, u, wl.elements, None)
    om = o.get_moments()
    assert max_abs(got[-1][outlets], om[outlets]) <= 4e-6
    assert max_abs(got[-1], om) <= 4e-6
    o.close()


@pytest.mark.parametrize("storage,nx,ny", [("f32", 64, 128), ("f16", 64, 128), ("bf16", 63, 127), ("f16", 95, 190)])
def test_pool_and_grid(cuda, storage, nx, ny):
    """The swimmer spans 0.25 nx to 0.25 nx + 0.4 ny: its tail beats next to the right outlet."""
    specs = [S.make_episode(nx, ny, seed=7, length=10), S.make_episode(ny, nx, seed=8, length=10)]
    pool = S.Pool(storage=storage, budget_bytes=256 << 20, max_episodes=4)
    slots = [pool.admit(sp) for sp in specs]
    envs = [S.PlainEnv(sp, storage) for sp in specs]
    for env in envs:
        env.g.profile(True, serial=True) # detection first
    for c in range(6):
        for k, (s, sp) in enumerate(zip(slots, specs)):
            a = np.random.default_rng(100 * c + k).uniform(-1, 1, 8).astype(np.float32)
            pool.set_action(s, a)
            envs[k].set_action(a)
        pool.advance()
        for s, env in zip(slots, envs):
            env.control_step(pool.substeps)
            assert pool.collect(s)[0].status == 0
            assert np.array_equal(pool.get_moments(s), env.g.get_moments()), f"control step {c}"
    for env in envs:
        env.close()
    pool.close()


@pytest.mark.parametrize("dim", [2, 3])
def test_more_outlets_than_faces_hold(cuda, dim):
    """Outlet nodes inside the grid, more than a list of the faces' size holds."""
    wl, rest = _scene2(64, 48) if dim == 2 else _scene3(40, 28, 30)
    f = wl.flags.reshape((wl.ny, wl.nx) if dim == 2 else (wl.nz, wl.ny, wl.nx)).copy()
    inner = f[..., 2:-2:3, 2:-2:2] if dim == 2 else f[2:-2, 2:-2, 2:-2:2]
    inner[inner == W.FLUID] = W.OUTLET_RIGHT
    wl.flags = f.reshape(-1)
    n = int((f[..., 1:] == W.OUTLET_RIGHT).sum())
    assert n > (2 * (64 + 48) if dim == 2 else 2 * (40 * 28 + 28 * 30 + 40 * 30))
    for storage in ("f32", "f16"):
        first, f0, _ = _states(wl, rest, storage, True, 5)
        beside, f1, _ = _states(wl, rest, storage, False, 5)
        assert all(np.array_equal(a, b) for a, b in zip(first, beside)) and np.array_equal(f0, f1)
        if storage == "f32":
            o = make_oracle(wl)
            for k in range(5):
                v, u = _surface(wl, rest, k)
                o.step(v, u, wl.elements, None)
            assert max_abs(beside[-1], o.get_moments()) <= 4e-6
            o.close()
