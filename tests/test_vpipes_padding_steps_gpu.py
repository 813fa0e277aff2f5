"""Whether a solve on rows that miss the TMA rules pads its state goes by its
steps, cells and outputs: the oracle's bits on both sides of each line, with
no output but z, with some and with all."""
import numpy as np
import pytest

from highmap_b200.inputs import fbm
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu
KW = dict(maintain_water_volume=0, dt=0.1, rain_per_step=1e-4, initial_water=0.0)


@pytest.mark.parametrize("outputs", [(), ("vel_u",), ("sediment", "vel_v"), ("water_depth", "sediment", "vel_u", "vel_v")])
@pytest.mark.parametrize("iters", [1, 2, 3, 5, 9, 20, 21])
@pytest.mark.parametrize("shape", [(24, 41), (70, 131), (259, 517)])
def test_steps_and_outputs(gpu, shape, iters, outputs):
    z0 = fbm(shape[1], shape[0], seed=45)
    want = dict(zip(("z", "water_depth", "sediment", "vel_u", "vel_v"),
                    po.vpipes(z0, po.VpipesParams.make(iterations=iters, **KW))))
    z = z0.copy()
    out = {name: np.empty_like(z) for name in outputs}
    gpu.hydraulic_vpipes(z, iterations=iters, **KW, **out)
    assert np.array_equal(z, want["z"])
    for name in outputs:
        assert np.array_equal(out[name], want[name]), name


@pytest.mark.parametrize("iters", [1, 2, 21])
@pytest.mark.parametrize("rain", [False, True])
def test_top_up(gpu, iters, rain):
    """(The sum's order differs from the oracle's: 1e-3 of the height range.)"""
    z0 = fbm(131, 70, seed=46)
    r = (0.25 + fbm(131, 70, seed=47)).astype(np.float32) if rain else None
    want = po.vpipes(z0, po.VpipesParams.make(iterations=iters), r)
    z, out = z0.copy(), [np.empty_like(z0) for _ in range(4)]
    gpu.hydraulic_vpipes(z, iterations=iters, rain_map=r, water_depth=out[0], sediment=out[1], vel_u=out[2], vel_v=out[3])
    for got, w in zip([z] + out, want):
        assert np.abs(got - w).max() <= 1e-3 * max(float(np.ptp(z0)), float(np.abs(w).max()))


@pytest.mark.parametrize("iters", [1, 2, 3])
@pytest.mark.parametrize("shape", [(24, 41), (300, 331), (400, 399)])
def test_flow(gpu, shape, iters):
    z, dm = fbm(shape[1], shape[0], seed=48), fbm(shape[1], shape[0], seed=49)
    assert np.array_equal(gpu.flow_simulation(z, 0.02, dm, iters), po.flow_simulation(z, 0.02, dm, iters))
