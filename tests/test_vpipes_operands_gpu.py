"""The square roots and quotients of the virtual-pipes step on random and
hard operands: grids of independent noise, every cell of its own magnitude,
so that a step takes millions of unrelated hypots, slopes and divisors; and
slopes whose hypot lies close to a rounding boundary.  Bit for bit against
the oracle, which rounds each from 64 bits or divides."""
import numpy as np
import pytest

from oracle import pyoracle as po

pytestmark = pytest.mark.gpu
KW = dict(maintain_water_volume=0, dt=0.1, k_capacity=0.05, k_erode=0.01, k_depose=0.01, evap_rate=0.01, gravity=9.81,
          rain_per_step=1e-4)
NAMES = ("z", "water", "sediment", "u", "v")


def _same(gpu, z0, rain, **kw):
    want = po.vpipes(z0, po.VpipesParams.make(**kw), rain)
    z = z0.copy()
    out = [np.empty_like(z) for _ in range(4)]
    gpu.hydraulic_vpipes(z, rain_map=rain, water_depth=out[0], sediment=out[1], vel_u=out[2], vel_v=out[3], **kw)
    for name, got, w in zip(NAMES, [z] + out, want):
        assert np.array_equal(got, w, equal_nan=True), name


@pytest.mark.parametrize("spread", [(-2, 0), (-6, 2), (-12, 6)])
@pytest.mark.parametrize("nx, ny", [(1540, 1300), (301, 160)])
def test_noise(gpu, nx, ny, spread):
    """(More than 2220 tiles: six CTAs per SM; under 296: a cell per thread.)"""
    rng = np.random.default_rng(nx - spread[0])
    z0 = (10.0 ** rng.uniform(*spread, (ny, nx))).astype(np.float32) * rng.choice(np.float32([-1, 1]), (ny, nx))
    rain = (10.0 ** rng.uniform(-3, 2, (ny, nx))).astype(np.float32)
    _same(gpu, z0.astype(np.float32), rain, iterations=3, initial_water=0.05, **KW)


@pytest.mark.parametrize("nx", [128, 300])
def test_slopes_at_rounding_boundaries(gpu, nx):
    """z = (p^2 - q^2, 2 p q) / 2 a column apart: the hypot is p^2 + q^2, or
    half way between two floats where that needs 25 bits, plus as little as
    the operands' last bit."""
    rng = np.random.default_rng(nx)
    ny = 420
    z0 = np.zeros((ny, nx), np.float32)
    for j in range(2, ny - 2, 4):
        for i in range(2, nx - 2, 4):
            p, q = rng.integers(2048, 5792, 2)
            a, b = np.float32(abs(p * p - q * q)), np.float32(2 * p * q)
            scale = np.float32(2.0 ** -int(rng.integers(20, 36)))
            # dz over the cell's neighbours: a along x, b along y
            z0[j, i + 1], z0[j + 1, i] = np.float32(2) * a * scale, np.float32(2) * b * scale
            if rng.random() < 0.3:
                z0[j, i + 1] = np.nextafter(z0[j, i + 1], np.float32(np.inf))
    _same(gpu, z0, None, iterations=1, initial_water=0.01, **KW)
    _same(gpu, z0, None, iterations=2, initial_water=0.0, **KW)
