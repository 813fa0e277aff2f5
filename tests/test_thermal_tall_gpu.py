"""Explicit steps per launch on grids with more rows than 65535 tiles, bit
for bit against the oracle."""
import numpy as np
import pytest

from highmap_b200.inputs import fbm
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


def _fields(nx, ny):
    z = np.tile(fbm(nx + 5, 4096, seed=91)[:, :nx], (ny // 4096 + 1, 1))[:ny].copy()
    z += np.linspace(0, 1, ny, dtype=np.float32)[:, None]
    t = np.full((ny, nx), 0.01, dtype=np.float32)
    return z, t


@pytest.mark.parametrize("time_block, rows, iters, nx, ny",
                         [(8, 0, 9, 3, 1100000), (2, 0, 2, 4, 1100000), (4, 0, 1, 3, 1100000), (6, 8, 6, 5, 300000),
                          (2, 128, 4, 3, 2000003), (8, 128, 8, 3, 1048560), (8, 128, 8, 6, 1048561)])
def test_more_rows_than_tiles(gpu, time_block, rows, iters, nx, ny):
    z0, t = _fields(nx, ny)
    want, want_d = po.thermal(z0, t, iters, deposition=True)
    gpu.thermal_set_launch(rows)
    try:
        z, d = z0.copy(), np.empty_like(z0)
        gpu.thermal(z, t, iters, deposition_map=d, time_block=time_block)
        assert np.array_equal(z, want) and np.array_equal(d, want_d)
        z = z0.copy()
        gpu.thermal(z, t, iters, time_block=time_block)
        assert np.array_equal(z, want)
    finally:
        gpu.thermal_set_launch(0)
