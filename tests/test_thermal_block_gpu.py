"""The several-steps-per-launch thermal kernel at the sizes where its tiles
can go wrong: grids of one tile and just over, odd widths, misaligned
buffers, every number of steps per launch, and cells the packed arithmetic
could treat differently (NaN heights, NaN, infinite and negative talus).
The bar is the one-step kernels': the oracle's bits."""
import numpy as np
import pytest

from highmap_b200.inputs import fbm
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


def _fields(nx, ny):
    z = fbm(nx, ny, seed=21)
    talus = ((0.5 + fbm(nx, ny, seed=22)) / max(nx, 8)).astype(np.float32)
    bed = (0.3 * z + 0.2 * fbm(nx, ny, seed=23)).astype(np.float32)
    return z, talus, bed


@pytest.mark.parametrize("time_block", [0, 2, 3, 5, 8])
@pytest.mark.parametrize("shape", [(3, 3), (4, 4), (5, 200), (200, 5), (16, 48), (17, 49), (20, 60), (28, 61),
                                   (33, 113), (129, 127)])
def test_tile_edges(gpu, shape, time_block):
    ny, nx = shape
    z0, talus, bed = _fields(nx, ny)
    for iters in (1, 2, 7, 16):
        want, want_d = po.thermal(z0, talus, iters, bedrock=bed, deposition=True)
        z, d = z0.copy(), np.empty_like(z0)
        gpu.thermal(z, talus, iters, bedrock=bed, deposition_map=d, time_block=time_block)
        assert np.array_equal(z, want) and np.array_equal(d, want_d)
        want, _ = po.thermal(z0, 0.5 / nx, iters)
        z = z0.copy()
        gpu.thermal(z, 0.5 / nx, iters, time_block=time_block)
        assert np.array_equal(z, want)


@pytest.mark.parametrize("mask", [False, True])
@pytest.mark.parametrize("iters", [0, 1, 9, 10])
def test_auto_bedrock_and_mask(gpu, iters, mask):
    z0, talus, _ = _fields(131, 70)
    m = fbm(131, 70, seed=24) if mask else None
    want, want_d = po.thermal_auto_bedrock(z0, talus, iters, deposition=True)
    if mask:  # the masked overload's blend, lerp(z0, result, mask)
        want = z0 * (np.float32(1) - m) + want * m
    z, d = z0.copy(), np.empty_like(z0)
    gpu.thermal_auto_bedrock(z, talus, iters, deposition_map=d, mask=m)
    assert np.array_equal(z, want) and np.array_equal(d, want_d)


def test_unusual_values(gpu):
    z0, talus, bed = _fields(90, 75)
    z0[10, 20] = z0[40, 63] = np.nan
    talus[5:9, 30:40] = np.nan
    talus[50:54, 10:14] = np.inf
    talus[60:64, 50:60] = -0.01
    talus[20, 20] = 0.0
    want, _ = po.thermal(z0, talus, 13, bedrock=bed)
    for tb in (0, 1, 4):
        z = z0.copy()
        gpu.thermal(z, talus, 13, bedrock=bed, time_block=tb)
        assert np.array_equal(z, want, equal_nan=True)


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("nx", [122, 123])
def test_buffer_alignment(gpu, offset, nx):
    import torch
    z0, talus, bed = _fields(nx, 50)
    want, _ = po.thermal(z0, talus, 11, bedrock=bed)

    def dev(x):
        t = torch.zeros(x.size + 1, device="cuda")[offset:offset + x.size].view(x.shape)
        t.copy_(torch.from_numpy(x))
        return t
    dz = dev(z0)
    gpu.thermal_device(dz, dev(talus), 11, bedrock=dev(bed))
    torch.cuda.synchronize()
    assert np.array_equal(dz.cpu().numpy(), want)


@pytest.mark.parametrize("rule", [0, 1, 2])
@pytest.mark.parametrize("shape", [(4, 4), (17, 49), (33, 113)])
def test_sibling_rules(gpu, rule, shape):
    ny, nx = shape
    z0, talus, _ = _fields(nx, ny)
    zmax = z0 + np.float32(0.25)
    f = (gpu.thermal_ridge, gpu.thermal_scree, gpu.thermal_schott)[rule]
    for iters in (1, 6, 13):
        want, want_d = po.thermal_sibling(rule, z0, talus, iters, zmax=zmax, deposition=True)
        z, d = z0.copy(), np.empty_like(z0)
        if rule == 1:
            f(z, talus, zmax, iters, deposition_map=d)
        else:
            f(z, talus, iters, deposition_map=d)
        assert np.array_equal(z, want) and np.array_equal(d, want_d)
