"""The D2Q9 dense pass's march units against the oracle at the sizes where a cut
can go wrong: remainders of the 64 columns and of the rows per unit, the
smallest grids, odd widths (cells fetched one by one), a solid that crosses
unit bounds and every storage.

A unit holds 64 columns and up to 14 rows; FFS_MARCH_ROWS pins the rows that a
grid's size would choose.  FP32 tolerances are those of test_gpu_random_flags.py: 4e-6
(a few units in the last place of density over the steps, bounce-back added
as a correction).  All D2Q9 cuts of a grid must give the same bits: the serving
pool cuts by its mix and must equal a grid stepped alone.
"""
import numpy as np
import pytest

from freeflow_b200 import workloads as W

from helpers import make_gpu, max_abs, run_pair

pytestmark = pytest.mark.gpu


def _random_walls(wl, seed, share=0.04):
    rng = np.random.default_rng(seed)
    f = wl.flags.copy()
    pick = (rng.random(f.size) < share) & (f == W.FLUID)
    f[pick] = rng.choice([W.WALL, W.SOLID, W.SOLID_DYNAMIC], size=int(pick.sum()))
    wl.flags = f
    return wl


def _box2(nx, ny, periodic, seed):
    wl = W.cylinder_channel_2d(nx=max(nx, 8), ny=max(ny, 8), radius=2.0, center=(3.0, 3.0), seed=seed)
    wl.nx, wl.ny = nx, ny
    rng = np.random.default_rng(seed)
    u = rng.uniform(-0.03, 0.03, (nx * ny, 2))
    wl.moments = W.equilibrium_moments(1.0 + rng.uniform(-1e-3, 1e-3, nx * ny), u)
    wl.flags = np.full(nx * ny, W.FLUID, np.uint8)
    if not periodic:
        f = wl.flags.reshape(ny, nx)
        f[0, :], f[-1, :], f[:, 0], f[:, -1] = W.WALL, W.OUTLET_UP, W.INLET_LEFT, W.OUTLET_RIGHT
    wl.elements, wl.periodic = None, 3 if periodic else 0
    return _random_walls(wl, seed)


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("nx,ny,rows", [(64, 14, 14), (65, 15, 14), (63, 29, 7), (128, 43, 14), (130, 17, 1), (2, 3, 1),
                                        (3, 2, 2), (127, 33, 13)])
def test_d2q9_cuts(cuda, monkeypatch, nx, ny, rows, periodic):
    monkeypatch.setenv("FFS_MARCH_ROWS", str(rows))
    gm, om, _, _, _ = run_pair(_box2(nx, ny, periodic, nx + ny), 4)
    assert max_abs(gm, om) <= 4e-6


@pytest.mark.parametrize("storage", ["f32", "f16", "bf16"])
def test_d2q9_cuts_round_identically(cuda, monkeypatch, storage):
    """A moving solid and outlets on four sides: the same bits for every cut."""
    wl = W.swimmer_2d(nx=150, ny=70, body_frac=0.5, n_boundary=80, seed=3)
    _same_bits(monkeypatch, wl, storage)


@pytest.mark.parametrize("storage", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("nx,ny,periodic", [(64, 32, False), (65, 33, True), (33, 9, False), (131, 75, False), (31, 7, True), (2, 3, False)])
def test_tiles_and_march_round_identically(cuda, monkeypatch, nx, ny, periodic, storage):
    """Walls and solids at random, an inlet and outlets, no surface."""
    _same_bits(monkeypatch, _box2(nx, ny, periodic, nx + 2 * ny), storage)


def _same_bits(monkeypatch, wl, storage):
    """Tiles, then the march with several rows per unit."""
    import torch

    out = []
    for rows in (None, "1", "5", "14"):
        if rows is None:
            monkeypatch.delenv("FFS_MARCH_ROWS", raising=False)
        else:
            monkeypatch.setenv("FFS_MARCH_ROWS", rows)
        g, s = make_gpu(wl, storage)
        for k in range(6):
            if s is not None:
                s.update(*wl.surface_at(k))
            g.step(s)
        torch.cuda.synchronize()
        assert g.status() == 0
        out.append((g.get_moments(), s.forces64.cpu().numpy() if s is not None else np.zeros(1)))
        g.close()
    for m, f in out[1:]:
        assert np.array_equal(out[0][0], m)
        assert np.array_equal(out[0][1], f)
