"""The stochastic rounding of 16-bit storage's velocity (binary16 in both
storages): a value goes to one of its two neighbours, upwards in magnitude with
the probability of its distance from the lower one, to within 2^-13 (13 random
bits), in binary16's normal and subnormal range, for either sign and each
component.  The random bits of neighbouring cells and of a cell's components
must be uncorrelated.  Statistical bounds are five standard deviations."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SU = 16.0  # velocities are stored as u * 16


def _stored(dim, storage, v):
    """Stored u * 16 of every cell for the same velocity (v in u * 16), densities of 128 values."""
    from freeflow_b200 import FluidGrid

    g = FluidGrid(dim=dim, nx=64, ny=64, nz=16 if dim == 3 else 1, fluid_viscosity=0.02, fluid_density=1.0,
                  fluid_dx=0.01, dt=0.01, storage=storage)
    m = np.zeros((g.ncell, g.nm), np.float32)
    m[:, 0] = 1.0 + np.random.default_rng(1).integers(-64, 64, g.ncell) / 1024.0
    m[:, 1:1 + dim] = np.float32(v / SU)
    g.set_moments(m)
    out = g.get_moments()[:, 1:1 + dim].astype(np.float64) * SU
    g.close()
    return out


@pytest.mark.parametrize("dim,storage", [(2, "f16"), (3, "f16"), (3, "bf16")])
@pytest.mark.parametrize("low", [0.0, 2.0 ** -24, 37 * 2.0 ** -24, 2.0 ** -14 - 2.0 ** -24, 2.0 ** -14, 2.0 ** -8, 1.5, 65472.0])
def test_neighbours_and_mean(cuda, low, dim, storage):
    ulp = max(2.0 ** (np.floor(np.log2(low)) - 10), 2.0 ** -24) if low else 2.0 ** -24
    for frac in (0.0, 0.125, 0.5, 0.875):
        for sign in (1.0, -1.0):
            u = sign * _stored(dim, storage, sign * (low + frac * ulp))
            assert np.isin(u, [low, low + ulp] if frac else [low]).all()
            up = (u - low) / ulp
            bound = 5.0 * np.sqrt(frac * (1.0 - frac) / len(u)) + 2.0 ** -13
            assert np.abs(up.mean(axis=0) - frac).max() <= bound


@pytest.mark.parametrize("frac", [0.25, 0.5])
def test_bits_are_uncorrelated(cuda, frac):
    up = (_stored(3, "f16", 0.5 + frac * 2.0 ** -11) - 0.5) * 2.0 ** 11
    up = (up - up.mean(axis=0)) / up.std(axis=0)
    n = len(up)
    for a in range(3):
        for b in range(a + 1, 3):
            assert abs((up[:, a] * up[:, b]).mean()) <= 5.0 / np.sqrt(n), (a, b)
        for step in (1, 2, 64, 64 * 64):     # the next cells in x, y and z
            assert abs((up[step:, a] * up[:-step, a]).mean()) <= 5.0 / np.sqrt(n - step), (a, step)
