"""Heights and talus at the ends of the float range, bit for bit against the
oracle: a no-data height of the type's lowest (or largest) value, infinite
heights, and talus that stops every exchange because it is infinite, NaN or
as large as a float can be.  The one-step sweeps and the kernel of several
steps per launch, with and without bedrock."""
import numpy as np
import pytest

from highmap_b200.inputs import fbm
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu
MAX = float(np.finfo(np.float32).max)
HEIGHTS = {"lowest": -MAX, "largest": MAX, "3e38": 3e38, "-3e38": -3e38, "-inf": -np.inf, "inf": np.inf}
TALUS = {"inf": np.inf, "nan": np.nan, "largest": MAX, "3e38": 3e38, "2.41e38": 2.41e38}
# (an infinite height only stays put where the talus is infinite or NaN)
CASES = [(h, t) for h in HEIGHTS for t in TALUS if "inf" not in h or t in ("inf", "nan")]


def _fields(nx, ny, height, talus):
    z = fbm(nx, ny, seed=81)
    t = ((0.5 + fbm(nx, ny, seed=82)) / nx).astype(np.float32)
    bed = (0.3 * z).astype(np.float32)
    z[10, 20] = z[11, 20] = z[30:34, 41:45] = np.float32(height)
    bed[10, 20] = bed[31:33, 42:44] = np.float32(height)
    t[8:14, 18:23] = t[28:36, 39:47] = np.float32(talus)
    return z, t, bed


@pytest.mark.parametrize("nx", [90, 91])
@pytest.mark.parametrize("height, talus", CASES)
def test_no_data_cells(gpu, height, talus, nx):
    z0, t, bed = _fields(nx, 75, HEIGHTS[height], TALUS[talus])
    for iters in (1, 4):
        for b in (None, bed):
            want, _ = po.thermal(z0, t, iters, bedrock=b)
            for tb in (0, 1, 2):
                z = z0.copy()
                gpu.thermal(z, t, iters, bedrock=b, time_block=tb)
                assert np.array_equal(z, want, equal_nan=True), (iters, b is None, tb)
        want, _ = po.thermal_auto_bedrock(z0, t, iters)
        z = z0.copy()
        gpu.thermal_auto_bedrock(z, t, iters)
        assert np.array_equal(z, want, equal_nan=True), iters


@pytest.mark.parametrize("talus", list(TALUS))
def test_uniform_talus(gpu, talus):
    z0, _, _ = _fields(90, 75, -MAX, 0.0)
    for iters in (1, 4):
        want, _ = po.thermal(z0, TALUS[talus], iters)
        z = z0.copy()
        gpu.thermal(z, TALUS[talus], iters)
        assert np.array_equal(z, want, equal_nan=True)
