"""Flow simulation with two steps per launch, bit for bit against the oracle:
grids at and around the smallest with blocked steps (40 x 24), tile edges,
every remainder of the row length, odd and even step counts; the last two
shapes have 364 and 665 tiles (256 and 512 threads per tile)."""
import numpy as np
import pytest

from highmap_b200.inputs import fbm
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("iters", [1, 2, 3, 8])
@pytest.mark.parametrize("shape", [(23, 40), (24, 39), (24, 40), (32, 64), (33, 65), (47, 66), (48, 67), (52, 100), (131, 237), (401, 419),
                                   (560, 606)])
def test_against_oracle(gpu, shape, iters):
    ny, nx = shape
    z, dm = fbm(nx, ny, seed=71), fbm(nx, ny, seed=72)
    for diffusion in (True, False):
        want = po.flow_simulation(z, 0.02, dm, iters, flux_diffusion=diffusion)
        assert np.array_equal(gpu.flow_simulation(z, 0.02, dm, iters, flux_diffusion=diffusion), want)
