"""The D3Q27 dense pass against the oracle, with 32-bit indices (grids of up to
429 M cells) and 64-bit ones (forced by FFS_DENSE3D_INDEX64), and cut into
chunks of planes at the depths where a cut can go wrong (FFS_DENSE3D_PLANES
pins the planes per chunk that a grid's size would choose).  FP32 grids take the
halo ring on two warps of its own, 16-bit ones on the tile's threads.
Tolerances are those of test_gpu_parity.py: 2e-6 against the ref32 oracle,
4e-6 next to walls (bounce-back added as a correction), 5e-6 against FP64.
"""
import numpy as np
import pytest

from freeflow_b200 import workloads as W

from helpers import make_gpu, max_abs, run_pair

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[32, 64], ids=lambda w: f"i{w}")
def index_width(request, monkeypatch):
    if request.param == 64:
        monkeypatch.setenv("FFS_DENSE3D_INDEX64", "1")
    return request.param


def test_swimmer(cuda, index_width):
    wl = W.swimmer_3d(nx=64, ny=32, nz=32, body_frac=0.3, nlat=12, nlon=16, seed=5)
    gm, om, gf, of, st = run_pair(wl, 6)
    assert st == 0
    assert max_abs(gm, om) <= 2e-6
    assert max_abs(gf, of) <= 1e-4 * np.abs(of).max()


def test_taylor_green_periodic_vs_fp64(cuda, index_width):
    wl = W.taylor_green_3d(n=32, u0=0.04, viscosity=0.005)
    gm, om, _, _, st = run_pair(wl, 20, precision="phys64")
    assert st == 0
    assert max_abs(gm, om) <= 5e-6


def test_reference_halo(cuda, index_width):
    """Non-periodic faces: the halo wraps at the low and clamps at the high face."""
    wl = W.taylor_green_3d(n=20, u0=0.04, viscosity=0.01)
    gm, om, _, _, st = run_pair(wl, 8, periodic=0)
    assert st == 0
    assert max_abs(gm, om) <= 2e-6


def test_walls_inlet_outlet(cuda, index_width):
    wl = W.swimmer_3d(nx=40, ny=24, nz=24, nlat=8, nlon=12)
    wl.elements = None
    gm, om, _, _, st = run_pair(wl, 8)
    assert st == 0
    assert max_abs(gm, om) <= 4e-6


def test_open_face_with_wall_across_the_wrap(cuda, index_width):
    wl = W.taylor_green_3d(n=20, u0=0.03, viscosity=0.01)
    f = wl.flags.reshape(20, 20, 20)
    f[:, :, 19] = W.WALL
    f[0, :, :] = W.WALL
    wl.flags = f.reshape(-1)
    gm, om, _, _, st = run_pair(wl, 6, periodic=0)
    assert st == 0
    assert max_abs(gm, om) <= 4e-6


@pytest.mark.parametrize("nz", [17, 40])
def test_odd_and_chunked_depths(cuda, index_width, nz):
    """Plane counts that leave a single plane in the last pair, and depths
    split into several z chunks."""
    wl = W.swimmer_3d(nx=48, ny=24, nz=nz, body_frac=0.3, nlat=8, nlon=12, seed=9)
    gm, om, _, _, st = run_pair(wl, 4)
    assert st == 0
    assert max_abs(gm, om) <= 4e-6


def test_periodic_width_not_a_tile_multiple(cuda, index_width):
    """nx = 48 with x periodic: the last tile's halo wraps onto the first
    columns, and its cells beyond nx only serve as halo."""
    wl = W.taylor_green_3d(n=48, u0=0.04, viscosity=0.01)
    nm = wl.moments.shape[1]
    wl.moments = np.ascontiguousarray(wl.moments.reshape(48, 48, 48, nm)[:12, :20, :].reshape(-1, nm))
    wl.flags = np.ascontiguousarray(wl.flags.reshape(48, 48, 48)[:12, :20, :].reshape(-1))
    wl.ny, wl.nz = 20, 12
    gm, om, _, _, st = run_pair(wl, 6)
    assert st == 0
    assert max_abs(gm, om) <= 2e-6


def test_odd_width(cuda, index_width):
    """nx odd: rows whose cells do not pair up on 8-byte boundaries."""
    wl = W.swimmer_3d(nx=41, ny=24, nz=20, body_frac=0.3, nlat=8, nlon=12, seed=11)
    gm, om, _, _, st = run_pair(wl, 4)
    assert st == 0
    assert max_abs(gm, om) <= 4e-6


@pytest.mark.parametrize("storage", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("nx,ny,nz", [(64, 32, 32), (45, 27, 23)])
def test_cuts_round_identically(cuda, monkeypatch, nx, ny, nz, storage):
    """The same bits (moments and surface forces, with walls, an inlet, an outlet
    and a moving surface) for every depth of a chunk and both index widths: the
    cut that a grid's size picks cannot change a result."""
    import torch

    wl = W.swimmer_3d(nx=nx, ny=ny, nz=nz, body_frac=0.4, nlat=16, nlon=24, seed=4)
    out = []
    for planes, wide in [(None, False), (1, False), (5, False), (nz, False), (None, True), (7, True)]:
        monkeypatch.delenv("FFS_DENSE3D_PLANES", raising=False)
        monkeypatch.setenv("FFS_DENSE3D_INDEX64", "1" if wide else "0")
        if planes:
            monkeypatch.setenv("FFS_DENSE3D_PLANES", str(planes))
        g, s = make_gpu(wl, storage)
        for k in range(6):
            s.update(*wl.surface_at(k))
            g.step(s)
        torch.cuda.synchronize()
        assert g.status() == 0
        out.append((g.get_moments(), s.forces64.cpu().numpy()))
        g.close()
    for o in out[1:]:
        assert np.array_equal(out[0][0], o[0])
        assert np.array_equal(out[0][1], o[1])


@pytest.mark.parametrize("planes", [1, 4, 19])
def test_cuts_random_node_types(cuda, monkeypatch, planes):
    """Walls, solids and moving-solid cells at random against the oracle, chunk by chunk."""
    from test_gpu_random_flags import _workload_3d

    monkeypatch.setenv("FFS_DENSE3D_PLANES", str(planes))
    gm, om, _, _, st = run_pair(_workload_3d(37, 21, 19, False, seed=5), 5)
    assert st == 0
    assert max_abs(gm, om) <= 4e-6
