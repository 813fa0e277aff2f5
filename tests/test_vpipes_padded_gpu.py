"""Virtual pipes and flow simulation on grids whose rows or buffers miss the
TMA rules: the state is kept in padded rows with a copy of z.  Sizes around
the smallest padded grid (40 x 24; 40 x 20 for the flow), every remainder
of the row length, misaligned device buffers, each output on its own.  The
bar is bit-exactness with the oracle (no volume top-up; with it, the sum's
order differs and the bar is 1e-3 of the height range)."""
import numpy as np
import pytest

from highmap_b200.inputs import fbm
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu
PKW = dict(maintain_water_volume=0, flux_diffusion=0, dt=0.1, k_capacity=0.05, k_erode=0.01, k_depose=0.01,
           evap_rate=0.01, gravity=9.81, rain_per_step=1e-4, initial_water=0.0)


def _want(z0, iters, rain=None, **kw):
    return po.vpipes(z0, po.VpipesParams.make(iterations=iters, **kw), rain)


@pytest.mark.parametrize("iters", [0, 1, 2, 9])
@pytest.mark.parametrize("shape", [(24, 41), (23, 41), (24, 39), (25, 42), (40, 43), (33, 131), (50, 129)])
def test_against_oracle(gpu, shape, iters):
    ny, nx = shape
    z0 = fbm(nx, ny, seed=41)
    rain = (0.5 + fbm(nx, ny, seed=42)).astype(np.float32)
    want = _want(z0, iters, rain, **PKW)
    z = z0.copy()
    out = [np.full_like(z, 7) for _ in range(4)]
    gpu.hydraulic_vpipes(z, iterations=iters, rain_map=rain, water_depth=out[0], sediment=out[1], vel_u=out[2],
                         vel_v=out[3], **PKW)
    for got, w in zip([z] + out, want):
        assert np.array_equal(got, w)


def test_top_up(gpu):
    z0 = fbm(125, 90, seed=43)
    want = _want(z0, 20)
    z, d = z0.copy(), np.empty_like(z0)
    gpu.hydraulic_vpipes(z, iterations=20, water_depth=d)
    assert np.abs(z - want[0]).max() <= 1e-3 and np.abs(d - want[1]).max() <= 1e-3


@pytest.mark.parametrize("which", ["vel_u", "vel_v", "sediment", "water_depth"])
@pytest.mark.parametrize("nx,offset", [(124, 1), (124, 2), (125, 0), (125, 1)])
def test_device_buffers_and_single_outputs(gpu, nx, offset, which):
    import torch
    z0 = fbm(nx, 60, seed=44)
    want = _want(z0, 7, **PKW)
    z = torch.zeros(z0.size + 2, device="cuda")[offset:offset + z0.size].view(z0.shape)
    z.copy_(torch.from_numpy(z0))
    o = torch.zeros(z0.size + 2, device="cuda")[offset:offset + z0.size].view(z0.shape)
    gpu.hydraulic_vpipes_device(z, gpu.vpipes_params(iterations=7, **PKW), **{which: o})
    torch.cuda.synchronize()
    assert np.array_equal(z.cpu().numpy(), want[0])
    assert np.array_equal(o.cpu().numpy(), want[{"water_depth": 1, "sediment": 2, "vel_u": 3, "vel_v": 4}[which]])


@pytest.mark.parametrize("iters", [0, 1, 6])
@pytest.mark.parametrize("shape", [(20, 41), (19, 41), (33, 131), (64, 66)])
def test_flow_simulation(gpu, shape, iters):
    ny, nx = shape
    z, dm = fbm(nx, ny, seed=45), fbm(nx, ny, seed=46)
    for dry in (0.0, 0.1):
        want = po.flow_simulation(z, 0.02, dm, iters, dry_out_ratio=dry)
        assert np.array_equal(gpu.flow_simulation(z, 0.02, dm, iters, dry_out_ratio=dry), want)
