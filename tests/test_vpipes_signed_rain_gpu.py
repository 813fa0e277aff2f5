"""The volume top-up with rain maps of either sign: it is add * rain / R with
R the map's sum, whatever R's sign and size.  Maps whose sum is negative
(zero-mean noise is half of the time), below the range of the reciprocal
that the tiles use, or both, plain and batched.  The sum's order differs
from the oracle's, so the bar is 1e-3: of the height range on z, of the
deepest water on the depth (a top-up of the wrong sign or size is off by
percents of the water per step)."""
import numpy as np
import pytest

from highmap_b200.inputs import fbm
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu
MAPS = {"negative": (-0.75, 1.0), "positive": (-0.25, 1.0), "tiny": (0.25, 1e-20), "tiny_negative": (-1.25, 1e-20),
        "large_negative": (-0.75, 1e25)}


def _case(nx, ny, name):
    shift, scale = MAPS[name]
    z0 = fbm(nx, ny, seed=71)
    rain = ((fbm(nx, ny, seed=72) + np.float32(shift)) * np.float32(scale)).astype(np.float32)
    assert name.endswith("negative") == (rain.sum(dtype=np.float64) < 0)
    return z0, rain


def _check(z, d, want, z0):
    assert np.isfinite(want[0]).all() and np.isfinite(want[1]).all()
    assert np.abs(z - want[0]).max() <= 1e-3 * float(np.ptp(z0))
    assert np.abs(d - want[1]).max() <= 1e-3 * float(np.abs(want[1]).max())


def _params(name, rps):
    # (a map of large values brings no more water than the others)
    return dict(iterations=5, dt=0.1, **(dict(initial_water=1e-27) if "large" in name else dict(rain_per_step=rps)))


@pytest.mark.parametrize("rps", [0.0, 1e-3])
@pytest.mark.parametrize("shape", [(64, 48), (37, 41), (240, 1028), (1040, 1028)])
@pytest.mark.parametrize("name", list(MAPS))
def test_plain(gpu, name, shape, rps):
    """(A cell per thread, padded rows, a pair per thread, and a grid whose
    top-up is summed between the steps.)"""
    z0, rain = _case(shape[1], shape[0], name)
    kw = _params(name, rps)
    want = po.vpipes(z0, po.VpipesParams.make(**kw), rain)
    z, d = z0.copy(), np.empty_like(z0)
    gpu.hydraulic_vpipes(z, rain_map=rain, water_depth=d, **kw)
    _check(z, d, want, z0)


@pytest.mark.parametrize("name", list(MAPS))
def test_batched(gpu, name):
    import torch
    from highmap_b200 import batch as B
    jobs, cases = [], []
    for nx, ny in ((64, 48), (131, 97)):
        z0, rain = _case(nx, ny, name)
        kw = _params(name, 0.0)
        z, r = torch.from_numpy(z0.copy()).cuda(), torch.from_numpy(rain).cuda()
        d = torch.empty_like(z)
        jobs.append(B.vpipes_job(z, rain_map=r, water_depth=d, **kw))
        cases.append((z, d, po.vpipes(z0, po.VpipesParams.make(**kw), rain), z0))
    B.run(jobs)
    torch.cuda.synchronize()
    for z, d, want, z0 in cases:
        _check(z.cpu().numpy(), d.cpu().numpy(), want, z0)
