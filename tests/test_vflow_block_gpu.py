"""The several-steps-per-launch viscous film kernel at the edges of its
tiles (44 x 22 outputs at five steps, wider at fewer), odd widths, and the
half-integer powers, which take a product and a square root instead of pow.
Tolerance: the function's own bar, 1e-3 of the deepest water; against fp64
powers the fp32 rounding of each face is the same except where the exact
power lies within 2^-50 of a rounding boundary."""
import numpy as np
import pytest

from highmap_b200.inputs import fbm
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu
TOL = 1e-3


def _close(got, want):
    assert float(np.abs(got.astype(np.float64) - want).max()) <= TOL * float(np.abs(want).max())


@pytest.mark.parametrize("iters", [1, 5, 6, 14, 21])
@pytest.mark.parametrize("shape", [(1, 1), (1, 45), (22, 44), (23, 45), (21, 87), (50, 131), (130, 88)])
def test_tile_edges(gpu, shape, iters):
    ny, nx = shape
    z = 0.1 * fbm(max(nx, 8), max(ny, 8), seed=31)[:ny, :nx].copy()
    dm = fbm(max(nx, 8), max(ny, 8), seed=32)[:ny, :nx].copy()
    for dry in (0.0, 0.1):
        _close(gpu.flow_simulation_viscous(z, 0.05, dm, iters, 0.5, dry),
               po.flow_simulation_viscous(z, 0.05, dm, iters, 0.5, dry))


@pytest.mark.parametrize("power", [1.0, 1.5, 2.0, 2.2, 2.5, 3.0, 3.5, 4.0, 0.5])
@pytest.mark.parametrize("viscosity", [1.0, 0.7])
def test_powers(gpu, power, viscosity):
    z = 0.1 * fbm(120, 90, seed=33)
    dm = fbm(120, 90, seed=34)
    _close(gpu.flow_simulation_viscous(z, 0.05, dm, 30, viscosity=viscosity, power=power),
           po.flow_simulation_viscous(z, 0.05, dm, 30, 0.5, 0.0, viscosity, power))


def test_large_grid_path(gpu):
    """Above 1.5 M cells each launch is one step: the same bits as two
    halves of the grid's own rule, here against the small-grid kernel on a
    band whose middle the band's edges cannot reach."""
    nx, ny, iters = 1300, 1200, 9
    z = 0.1 * fbm(nx, ny, seed=35)
    dm = fbm(nx, ny, seed=36)
    dm[600, 600] = 1.5  # the deepest cell, in the band: both runs take the same time step
    full = gpu.flow_simulation_viscous(z, 0.05, dm, iters)
    band = gpu.flow_simulation_viscous(z[500:700].copy(), 0.05, dm[500:700].copy(), iters)
    assert np.array_equal(full[500 + iters:700 - iters], band[iters:200 - iters])
