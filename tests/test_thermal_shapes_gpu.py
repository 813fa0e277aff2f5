"""Grids of a few rows or columns, where the choice between one and several
steps per launch goes by how the shape fills the tiles: the oracle's bits on
both sides of it, for the exchange and for a sibling stencil."""
import numpy as np
import pytest

from highmap_b200.inputs import fbm
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("iters", [2, 5, 10])
@pytest.mark.parametrize("nx, ny", [(3, 60000), (4, 60001), (30000, 4), (30001, 5), (20000, 17), (4, 150001), (64, 9000), (61, 9000)])
def test_thin_grids(gpu, nx, ny, iters):
    w, h = min(nx, 512), min(ny, 512)
    z0 = np.tile(fbm(max(w, 8), max(h, 8), seed=41)[:h, :w], (ny // h + 1, nx // w + 1))[:ny, :nx].copy()
    t = np.full_like(z0, 0.02)
    want, want_d = po.thermal(z0, t, iters, bedrock=0.5 * z0, deposition=True)
    z, d = z0.copy(), np.empty_like(z0)
    gpu.thermal(z, t, iters, bedrock=0.5 * z0, deposition_map=d)
    assert np.array_equal(z, want) and np.array_equal(d, want_d)
    want, _ = po.thermal_sibling(0, z0, t, iters)
    z = z0.copy()
    gpu.thermal_ridge(z, t, iters)
    assert np.array_equal(z, want)
