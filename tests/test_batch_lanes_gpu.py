"""Batches of more than a few milliseconds of work, whose thermal jobs and
larger virtual-pipes jobs run on four side streams: every job gives the bits
of its plain call, and a virtual-pipes job whose tile loads time out there
makes the run report it."""
import numpy as np
import pytest

from highmap_b200 import _lib as L
from highmap_b200.inputs import fbm

pytestmark = pytest.mark.gpu
RAIN = dict(maintain_water_volume=0, dt=0.1, rain_per_step=1e-4, initial_water=0.0)


def _dev(a, offset=0):
    import torch
    t = torch.zeros(a.size + offset, device="cuda")[offset:].view(a.shape)
    t.copy_(torch.from_numpy(a))
    return t


def _specs():
    """(kind, nx, ny, iterations, options, floats off 16 bytes): over 4 ms
    of work; virtual-pipes jobs above 2^17 cells on the lanes (aligned and
    padded), below in the rounds; thermal jobs of all sizes on the lanes."""
    return [("thermal", 1024, 1024, 1100, dict(bedrock=True), 0),
            ("thermal", 1031, 700, 60, dict(depo=True), 1),
            ("thermal", 65, 48, 30, dict(depo=True), 0),
            ("thermal", 4, 3, 9, dict(), 0),
            ("vpipes", 512, 256, 40, dict(), 0),
            ("vpipes", 517, 259, 35, dict(maps=True), 0),
            ("vpipes", 512, 300, 30, RAIN, 1),
            ("vpipes", 1025, 1024, 9, dict(maps=True, **RAIN), 0),
            ("vpipes", 700, 190, 25, dict(pipe_length=2.0), 0),
            ("vpipes", 130, 120, 33, dict(maps=True), 0),
            ("vpipes", 131, 97, 33, RAIN, 1)]


def _make(specs, seed=0):
    import torch
    out = []
    for k, (kind, nx, ny, it, o, off) in enumerate(specs):
        o = dict(o)
        z = _dev(fbm(max(nx, 8), max(ny, 8), seed=seed + k)[:ny, :nx].copy(), off)
        extra = {}
        if kind == "thermal":
            extra["talus"] = _dev(((0.5 + fbm(nx, ny, seed=50 + k)) / nx).astype(np.float32))
            if o.get("bedrock"):
                extra["bedrock"] = 0.3 * z
            if o.get("depo"):
                extra["deposition_map"] = torch.empty_like(z)
        else:
            if o.pop("maps", False):
                extra["rain_map"] = _dev((0.2 + fbm(nx, ny, seed=60 + k)).astype(np.float32))
            for name in ("water_depth", "sediment", "vel_u", "vel_v"):
                extra[name] = torch.empty_like(z)
            extra["params"] = o
        out.append((kind, z, it, extra))
    return out


def _job(kind, z, it, extra):
    from highmap_b200 import batch as B
    e = dict(extra)
    if kind == "thermal":
        return B.thermal_job(z, e.pop("talus"), it, **e)
    return B.vpipes_job(z, it, **e.pop("params"), **e)


def _plain(gpu, kind, z, it, extra):
    e = dict(extra)
    if kind == "thermal":
        gpu.thermal_device(z, e.pop("talus"), it, **e)
    else:
        gpu.hydraulic_vpipes_device(z, gpu.vpipes_params(iterations=it, **e.pop("params")), **e)


OUTPUTS = ("deposition_map", "water_depth", "sediment", "vel_u", "vel_v")


@pytest.mark.parametrize("use_graph", [True, False])
def test_jobs_equal_plain_calls(gpu, use_graph):
    import torch
    from highmap_b200 import batch as B
    got, want = _make(_specs()), _make(_specs())
    for c in want:
        _plain(gpu, *c)
    B.run([_job(*c) for c in got], use_graph=use_graph)
    torch.cuda.synchronize()
    for g, w, s in zip(got, want, _specs()):
        assert torch.equal(g[1], w[1]), s
        for name in OUTPUTS:
            if name in g[3]:
                assert torch.equal(g[3][name], w[3][name]), (s, name)


def test_kernel_choice_changes_meanwhile(gpu):
    """Another thread changes the process's choice of step kernels, which
    decides whether a job's rows are padded, while batches run: a lane's
    scratch fits what its jobs then do, and the bits stay."""
    import threading
    import torch
    from highmap_b200 import batch as B
    specs = [("vpipes", 517, 259 + k, 12, RAIN, k % 2) for k in range(12)] + [("thermal", 1024, 1024, 1300, dict(), 0)]
    want = _make(specs)
    for c in want:
        _plain(gpu, *c)
    stop = threading.Event()

    def flip():
        while not stop.is_set():
            for algo in (gpu.VPIPES_TILED_CP_ASYNC, gpu.VPIPES_TILED):
                gpu.vpipes_set_algorithm(algo)

    t = threading.Thread(target=flip)
    t.start()
    try:
        for _ in range(10):
            got = _make(specs)
            B.run([_job(*c) for c in got], use_graph=False)
            torch.cuda.synchronize()
            for g, w, s in zip(got, want, specs):
                assert torch.equal(g[1], w[1]), s
    finally:
        stop.set()
        t.join()
        gpu.vpipes_set_algorithm(gpu.VPIPES_AUTO)


@pytest.mark.parametrize("use_graph", [True, False])
@pytest.mark.parametrize("first", [0, 1])
def test_lane_timeout_is_reported(gpu, use_graph, first):
    """The test hook makes every TMA tile's bounded wait run out; a later job
    on the same lane starts with a clean error word and may be shorter or a
    thermal one."""
    import torch
    from highmap_b200 import batch as B
    specs = [("thermal", 1024, 1024, 1200, dict(), 0), ("vpipes", 512, 256, 1, RAIN, 0), ("vpipes", 64, 48, 2, RAIN, 0)]
    if first:
        specs = specs[1:]
        specs[0] = ("vpipes", 1024, 1024, 1, RAIN, 0)  # above 2^20 cells: the one lane of smaller batches
    jobs = [_job(*c) for c in _make(specs)]
    try:
        gpu.vpipes_set_algorithm(gpu.VPIPES_TILED)
        gpu.debug_tma_expect_extra(16)
        with pytest.raises(L.HMError) as e:
            B.run(jobs, use_graph=use_graph)
        assert e.value.status == L.HM_ERR_TIMEOUT and "timed out" in str(e.value)
    finally:
        gpu.debug_tma_expect_extra(0)
        gpu.vpipes_set_algorithm(gpu.VPIPES_AUTO)
    got, want = _make(specs), _make(specs)
    B.run([_job(*c) for c in got], use_graph=use_graph)
    for c in want:
        _plain(gpu, *c)
    torch.cuda.synchronize()
    for g, w in zip(got, want):
        assert torch.equal(g[1], w[1])
