"""A NaN in the initial depth of the viscous film.  The reference's maximum
starts at the first cell and takes what compares greater, so a NaN counts
only there; elsewhere it is passed over.  A step turns it into dry ground.
Tolerance: the function's own bar, 1e-3 of the deepest water."""
import numpy as np
import pytest

from highmap_b200.inputs import fbm
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("power", [2.5, 2.2, 2.0])
@pytest.mark.parametrize("cells", [[(0, 0)], [(20, 21)], [(0, 0), (20, 21)], [(0, 1)], [(1, 0)], [(39, 63)]])
def test_nan_depth(gpu, cells, power):
    z = 0.1 * fbm(64, 40, seed=37)
    for sign in (1.0, -1.0):
        dm = fbm(64, 40, seed=38)
        for c in cells:
            dm[c] = np.copysign(np.float32("nan"), np.float32(sign))
        for iters in (0, 1, 12):
            for dry in (0.0, 0.1):
                want = po.flow_simulation_viscous(z, 0.05, dm, iters, 0.5, dry, 1.0, power)
                got = gpu.flow_simulation_viscous(z, 0.05, dm, iters, 0.5, dry, power=power)
                assert np.array_equal(np.isnan(got), np.isnan(want))
                ok = ~np.isnan(want)
                assert np.abs(got[ok].astype(np.float64) - want[ok]).max() <= 1e-3 * np.abs(want[ok]).max()
