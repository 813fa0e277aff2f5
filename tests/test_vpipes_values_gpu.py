"""The tiled virtual-pipes step evaluates pairs of cells in packed fp32
arithmetic, with square roots and quotients that fall back to the exact
forms outside the range they are proven for.  Values inside, at the edge of
and outside that range, bit for bit against the oracle: water from almost
nothing to deeper than the relief, relief from flat to 1e15, dry basins,
floors at the smallest scale; with and without flux diffusion."""
import numpy as np
import pytest

from highmap_b200.inputs import fbm
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu
BASE = dict(maintain_water_volume=0, dt=0.1, k_capacity=0.05, k_erode=0.01, k_depose=0.01, evap_rate=0.01,
            gravity=9.81, rain_per_step=1e-4, initial_water=0.0, iterations=8)
CASES = {
    "ordinary": (1.0, {}),
    "steep": (1e6, {}),
    "huge": (1e15, {}),
    "flat": (0.0, {}),
    "shallow": (1e-12, {}),
    "film": (1.0, dict(rain_per_step=0.0, initial_water=1e-25)),
    "vanishing": (1.0, dict(rain_per_step=0.0, initial_water=1e-38)),
    "deep": (1.0, dict(initial_water=1e3)),
    "low_floor": (1.0, dict(water_height=1e-6)),
    "film_low_floor": (1.0, dict(water_height=1e-14, rain_per_step=0.0, initial_water=1e-25)),
    "high_floor": (1.0, dict(water_height=1e25)),
}


@pytest.mark.parametrize("diffusion", [0, 1])
@pytest.mark.parametrize("nx", [128, 131, 2084])
@pytest.mark.parametrize("case", list(CASES))
def test_magnitudes(gpu, case, nx, diffusion):
    """(Grids of up to 296 tiles of 32 x 16 run a cell per thread, larger
    ones a pair.)"""
    scale, extra = CASES[case]
    z0 = (fbm(nx, 70, seed=51) * np.float32(scale)).astype(np.float32)
    z0[20:30, 40:60] = z0.min()  # a dry, then filling, flat basin
    kw = {**BASE, "flux_diffusion": diffusion, **extra}
    want = po.vpipes(z0, po.VpipesParams.make(**kw))
    z = z0.copy()
    out = [np.empty_like(z) for _ in range(4)]
    gpu.hydraulic_vpipes(z, water_depth=out[0], sediment=out[1], vel_u=out[2], vel_v=out[3], **kw)
    for name, got, w in zip(("z", "water", "sediment", "u", "v"), [z] + out, want):
        assert np.array_equal(got, w), name


@pytest.mark.parametrize("diffusion", [0, 1])
@pytest.mark.parametrize("nx", [1028, 1031])
def test_many_tiles(gpu, nx, diffusion):
    """More than 2220 tiles: six CTAs per SM."""
    z0 = fbm(nx, 1090, seed=52)
    kw = {**BASE, "flux_diffusion": diffusion, "iterations": 4}
    want = po.vpipes(z0, po.VpipesParams.make(**kw))
    z = z0.copy()
    out = [np.empty_like(z) for _ in range(4)]
    gpu.hydraulic_vpipes(z, water_depth=out[0], sediment=out[1], vel_u=out[2], vel_v=out[3], **kw)
    for name, got, w in zip(("z", "water", "sediment", "u", "v"), [z] + out, want):
        assert np.array_equal(got, w), name
