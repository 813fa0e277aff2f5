"""The flow-only tiles' wait for their TMA boxes is bounded too, and running
out is reported with the caller's output untouched: the test hook arms every
tile's barrier with bytes that never come.  One step runs the one-step
kernel, two the two-step one, three both; with rows of a multiple of 4
floats and padded (which one step is from 100000 cells on)."""
import numpy as np
import pytest

from highmap_b200 import _lib as L
from highmap_b200.inputs import fbm
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("iters", [1, 2, 3])
@pytest.mark.parametrize("nx, ny", [(64, 40), (67, 1500)])
def test_wait_runs_out_and_is_reported(gpu, nx, ny, iters):
    import ctypes as C
    z, dm = fbm(nx, ny, seed=13), fbm(nx, ny, seed=14)
    out = np.full_like(z, -7.0)
    ctx = gpu.Context(0)

    def p(a):
        return C.c_void_p(a.ctypes.data)

    def call():
        return L.lib().hm_flow_simulation(ctx.handle, p(z), nx, ny, C.c_float(0.05), p(dm), iters, C.c_float(0.5), 1,
                                          C.c_float(0.01), C.c_float(0.0), p(out))
    try:
        gpu.debug_tma_expect_extra(16)
        assert call() == L.HM_ERR_TIMEOUT
        assert (out == -7.0).all()
    finally:
        gpu.debug_tma_expect_extra(0)
    assert call() == 0
    ctx.close()
    assert np.array_equal(out, po.flow_simulation(z, 0.05, dm, iters, 0.5, True, 0.01, 0.0))
