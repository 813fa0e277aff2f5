"""The viscous film's mobilities h^power are rounded once from 64 bits: one
step against a NumPy restatement that forms each power in float64, rounds
it, and keeps the step's fp32 operations and their order, bit for bit.
Powers that are products and square roots, and depths at zero, inside and
outside the range in which a half power is taken from fp32 pairs.  (A
float64 pow is off by at most 2^-52 of the power; depths whose power lies
within 2^-50 of a rounding boundary are left out.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
F = np.float32


def _pow(x, power):
    """x^power rounded to float32 from extended precision."""
    x = x.astype(np.longdouble)
    r = np.ones_like(x)
    for _ in range(int(power)):
        r = r * x
    return (r * np.sqrt(x) if power % 1 else r).astype(F)


def _clear_of_boundaries(x, power):
    """where float64 and float32 roundings of x^power agree whatever the
    last bits of the float64 power"""
    p = x.astype(np.float64) ** power
    with np.errstate(all="ignore"):
        return ((p * (1 + 2.0 ** -50)).astype(F) == (p * (1 - 2.0 ** -50)).astype(F)) | (p == 0)


def _step(z, h, power):
    """The first step, viscosity 1; and where its rounding is certain."""
    hp, zp = np.pad(h, 1, mode="edge"), np.pad(z, 1, mode="edge")
    c = (slice(1, -1), slice(1, -1))
    at = {"e": (slice(1, -1), slice(2, None)), "w": (slice(1, -1), slice(None, -2)), "n": (slice(2, None), slice(1, -1)),
          "s": (slice(None, -2), slice(1, -1))}
    H = hp + zp
    sure = np.ones(h.shape, bool)
    M = {}
    for k, a in at.items():
        m = F(0.5) * (hp[c] + hp[a])
        sure &= _clear_of_boundaries(m, power)
        M[k] = _pow(m, power)
    q = {"e": -M["e"] * (H[at["e"]] - H[c]), "w": -M["w"] * (H[c] - H[at["w"]]),
         "n": -M["n"] * (H[at["n"]] - H[c]), "s": -M["s"] * (H[c] - H[at["s"]])}
    dhdt = -(((q["e"] - q["w"]) + q["n"]) - q["s"])
    dt = F(0.2) / np.maximum(_pow(h.max()[None], power)[0], F(1e-6))
    return np.maximum(F(0), h + dt * dhdt), sure


@pytest.mark.parametrize("scale", [1.0, 1e-3, 3e-8, 1e-8, 3e-9, 1e-12, 1e4, 9e7, 3e8])
@pytest.mark.parametrize("power", [1.0, 1.5, 2.0, 2.5, 3.0, 3.5, 4.0])
def test_one_step(gpu, power, scale):
    if scale ** (power + 1) > 2e38:
        scale = 1e7  # (the fluxes would overflow)
    rng = np.random.default_rng(int(power * 10))
    h = (rng.random((400, 700), dtype=F) ** 3 * F(scale)).astype(F)
    h[rng.random(h.shape) < 0.05] = 0
    h[200:210, 300:340] = 0
    z = (rng.random(h.shape, dtype=F) * F(scale)).astype(F)
    # the same cells in a tile kernel and, above 1.5 M cells, in the one-step one
    for rows in (400, 2200):
        hh, zz = (np.tile(a, (rows // 400 + 1, 1))[:rows].copy() for a in (h, z))
        want, sure = _step(zz, hh, power)
        got = gpu.flow_simulation_viscous(zz, 1.0, hh, 1, power=power)
        assert sure.mean() > 0.999
        assert np.array_equal(got[sure], want[sure])
