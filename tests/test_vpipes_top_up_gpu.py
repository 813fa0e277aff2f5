"""The volume top-up on grids around the size from which one CTA sums the
tiles' water between two steps (above 2048 tiles of 32 x 16) instead of
every tile for itself.  The sum's order differs from the oracle's, so the
bar is 1e-3 of the height range on z, sediment and water depth."""
import numpy as np
import pytest

from highmap_b200.inputs import fbm
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


def _run(gpu, z0, iters, rain):
    want = po.vpipes(z0, po.VpipesParams.make(iterations=iters), rain)
    z, d, s = z0.copy(), np.empty_like(z0), np.empty_like(z0)
    gpu.hydraulic_vpipes(z, iterations=iters, rain_map=rain, water_depth=d, sediment=s)
    for got, w in zip((z, d, s), want):
        assert np.isfinite(got).all() and np.abs(got - w).max() <= 1e-3 * float(np.ptp(z0))


@pytest.mark.parametrize("iters", [1, 2, 5])
@pytest.mark.parametrize("with_rain", [False, True])
@pytest.mark.parametrize("shape", [(1024, 1024), (1025, 1024), (1040, 1021), (16, 65568)])
def test_tile_counts(gpu, shape, with_rain, iters):
    z0 = fbm(shape[1], shape[0], seed=61)
    _run(gpu, z0, iters, (0.25 + fbm(shape[1], shape[0], seed=62)).astype(np.float32) if with_rain else None)


@pytest.mark.parametrize("shape", [(20, 44), (37, 41), (64, 100), (33, 1028)])
@pytest.mark.parametrize("rps", [0.0, 1e-3])
def test_rain_maps(gpu, shape, rps):
    """Zeros, faint and heavy rain in one map, which the tiles stage with
    their ring clamped to the grid; aligned and padded rows."""
    z0 = fbm(shape[1], shape[0], seed=63)
    rain = fbm(shape[1], shape[0], seed=64)
    rain = np.where(rain < 0.3, 0, np.where(rain < 0.5, 1e-25, np.where(rain > 0.8, 50, rain))).astype(np.float32)
    want = po.vpipes(z0, po.VpipesParams.make(iterations=9, rain_per_step=rps), rain)
    z, d = z0.copy(), np.empty_like(z0)
    gpu.hydraulic_vpipes(z, iterations=9, rain_map=rain, rain_per_step=rps, water_depth=d)
    assert np.abs(z - want[0]).max() <= 1e-3 * float(np.ptp(z0))
    assert np.abs(d - want[1]).max() <= 1e-3 * max(float(np.ptp(z0)), float(want[1].max()))
