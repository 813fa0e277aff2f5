"""A NaN water height with a given initial water: the reference's max takes
the depth itself as the velocity's divisor and the depth ratio at its cap,
so z stays finite where the water moves.  Bit for bit against the oracle."""
import numpy as np
import pytest

from highmap_b200.inputs import fbm
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("algo", [0, 1, 2])
@pytest.mark.parametrize("nx", [64, 67, 2084])
def test_nan_water_height(gpu, nx, algo):
    z0 = fbm(nx, 70, seed=53)
    kw = dict(water_height=float("nan"), maintain_water_volume=0, dt=0.1, rain_per_step=1e-4, initial_water=0.01,
              iterations=4)
    want = po.vpipes(z0, po.VpipesParams.make(**kw))
    z = z0.copy()
    out = [np.empty_like(z) for _ in range(4)]
    gpu.vpipes_set_algorithm(algo)
    try:
        gpu.hydraulic_vpipes(z, water_depth=out[0], sediment=out[1], vel_u=out[2], vel_v=out[3], **kw)
    finally:
        gpu.vpipes_set_algorithm(gpu.VPIPES_AUTO)
    for name, got, w in zip(("z", "water", "sediment", "u", "v"), [z] + out, want):
        assert np.array_equal(got, w, equal_nan=True), name
    assert np.isfinite(want[0]).mean() > 0.5
