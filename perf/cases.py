"""What is measured: calls a program makes to this library, from the
smallest to the largest, through the public entry points.

The two solvers, thermal erosion and virtual-pipes hydraulic erosion, are
called on host heightmaps (numpy arrays, as HighMap's own functions take
``hmap::Array``), on grids that stay on the device (a terrain pipeline that
chains calls) and as a batch of many heightmaps.  The callers and relatives
that share their kernels follow: auto-bedrock thermal erosion, flow
simulation, sediment deposition, the talus stencils and the viscous film.

Sizes are those of this repository's tests and benchmark (256^2 with 100
iterations, 4096^2, the default 10 and 50 iterations, mixed batches) and
the odd and ragged sizes terrain grids come in (2^k + 1 heightfields, crops).
The solvers update the heights in place, so a pass first copies the kept
input heights into the working grid, as a program that keeps its input does.
"""
import math

import numpy as np
import torch

from highmap_b200 import batch as B
from highmap_b200 import gpu as G

# virtual-pipes parameters of the 4096^2 benchmark (rain every step, no
# volume top-up); the other calls take the function's defaults
RAIN = dict(maintain_water_volume=0, flux_diffusion=0, dt=0.1, k_capacity=0.05, k_erode=0.01, k_depose=0.01,
            evap_rate=0.01, gravity=9.81, pipe_area=1.0, pipe_length=1.0, rain_per_step=1e-4, initial_water=0.0,
            water_height=1e-2)
DEFAULTS = dict(maintain_water_volume=1, flux_diffusion=1, dt=0.5, k_capacity=0.5, k_erode=0.001, k_depose=0.01,
                evap_rate=0.1, gravity=1.0, pipe_area=1.0, pipe_length=1.0, rain_per_step=0.0, initial_water=-1.0,
                water_height=1e-2)
STENCILS = {"ridge": G.RIDGE, "scree": G.SCREE, "inflate": G.INFLATE, "rib": G.RIB}


# ------------------------------------------------------------------ cases

def listed():
    return [
        # the reference configuration of thermal erosion: one small host
        # heightmap, uniform talus, deposition map wanted
        dict(name="thermal_256_host", kind="thermal", host=True, nx=256, ny=256, iterations=100, talus="value",
             bedrock=False, deposition=True, mask=False, auto=False),
        # a 2^k + 1 tile settled with the default 10 iterations, every
        # optional grid of the call in use: the shortest call of the list
        dict(name="thermal_513x257", kind="thermal", host=False, nx=513, ny=257, iterations=10, talus="map",
             bedrock=True, deposition=True, mask=True, auto=False),
        # the benchmark's thermal solve: talus map and bedrock, full length
        dict(name="thermal_4096", kind="thermal", host=False, nx=4096, ny=4096, iterations=500, talus="map",
             bedrock=True, deposition=False, mask=False, auto=False),
        # a mid-size terrain with uniform talus and the self-built bedrock
        dict(name="auto_bedrock_2048", kind="thermal", host=False, nx=2048, ny=2048, iterations=100, talus="value",
             bedrock=False, deposition=True, mask=False, auto=True),
        # an editor node on a small host heightmap, defaults, all outputs
        dict(name="vpipes_256_host", kind="vpipes", host=True, nx=256, ny=256, iterations=50, preset="defaults",
             rain_map=False, outputs=True),
        # a ragged crop with a rain map, defaults, all outputs
        dict(name="vpipes_1023x767", kind="vpipes", host=False, nx=1023, ny=767, iterations=50, preset="defaults",
             rain_map=True, outputs=True),
        # the benchmark's hydraulic solve (its size-sweep length)
        dict(name="vpipes_4096", kind="vpipes", host=False, nx=4096, ny=4096, iterations=200, preset="rain",
             rain_map=False, outputs=False),
        # water routing over a fixed terrain
        dict(name="flow_1024", kind="flow", nx=1024, ny=1024, iterations=200, dry_out=0.01),
        # a viscous film, default power
        dict(name="viscous_512", kind="viscous", nx=512, ny=512, iterations=200, power=2.5),
        # sediment laid down in the default 5 layers of 10 settling steps
        dict(name="deposition_1024", kind="deposition", nx=1024, ny=1024, layers=5, iterations=10),
        # a sibling talus rule on a 2^k + 1 heightfield
        dict(name="ridge_1025", kind="stencil", rule="ridge", nx=1025, ny=1025, iterations=50),
        # many heightmaps of uneven sizes and lengths in one batch
        dict(name="batch_48", kind="batch", jobs=48, lo=128, hi=1024, iterations=200, jobseed=7),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _side(rng, lo, hi):
    """A grid side: log-uniform, left as it falls (odd as often as even),
    rounded to a multiple of 8, or a 2^k + 1 heightfield's."""
    s = int(round(_log(rng, lo, hi)))
    form = rng.randrange(4)
    if form == 0:
        s = 8 * max(1, round(s / 8))
    elif form == 1:
        s = 2 ** int(round(math.log2(s))) + rng.randrange(2)
    return max(lo, min(hi, s))


def _sides(rng, lo, hi):
    a = _side(rng, lo, hi)
    if rng.random() < 0.4:
        return a, a
    b = max(lo, min(hi, int(round(a / rng.uniform(1.0, 2.0)))))
    return (a, b) if rng.random() < 0.5 else (b, a)


def _iters(rng, lo, hi, nx, ny, budget):
    """Log-uniform iterations, at most `budget` cell-updates."""
    return max(lo, min(int(round(_log(rng, lo, hi))), int(budget // (nx * ny))))


def draw(rng):
    kind = rng.choice(["thermal", "thermal", "thermal", "vpipes", "vpipes", "vpipes", "flow", "viscous", "deposition",
                       "stencil", "batch"])
    if kind == "thermal":
        host = rng.random() < 0.3
        nx, ny = _sides(rng, 64, 2048 if host else 4096)
        auto = rng.random() < 0.25
        return dict(kind=kind, host=host, nx=nx, ny=ny, iterations=_iters(rng, 5, 500, nx, ny, 3e9),
                    talus=rng.choice(["map", "value"]), bedrock=not auto and rng.random() < 0.5,
                    deposition=rng.random() < 0.5, mask=rng.random() < 0.3, auto=auto)
    if kind == "vpipes":
        host = rng.random() < 0.3
        nx, ny = _sides(rng, 64, 2048 if host else 4096)
        return dict(kind=kind, host=host, nx=nx, ny=ny, iterations=_iters(rng, 10, 500, nx, ny, 1.5e9),
                    preset=rng.choice(["defaults", "rain"]), rain_map=rng.random() < 0.4, outputs=rng.random() < 0.6)
    if kind == "batch":
        return dict(kind=kind, jobs=int(round(_log(rng, 8, 64))), lo=128, hi=1024,
                    iterations=int(round(_log(rng, 50, 200))), jobseed=rng.randrange(10 ** 6))
    nx, ny = _sides(rng, 96, 2048)
    if kind == "flow":
        return dict(kind=kind, nx=nx, ny=ny, iterations=_iters(rng, 20, 500, nx, ny, 1.5e9),
                    dry_out=rng.choice([0.0, 0.01]))
    if kind == "viscous":
        return dict(kind=kind, nx=nx, ny=ny, iterations=_iters(rng, 20, 400, nx, ny, 6e8),
                    power=rng.choice([2.5, 2.5, 3.0, 2.2]))
    if kind == "deposition":
        return dict(kind=kind, nx=nx, ny=ny, layers=rng.randrange(3, 12), iterations=_iters(rng, 5, 40, nx, ny, 2e8))
    return dict(kind=kind, rule=rng.choice(sorted(STENCILS)), nx=nx, ny=ny,
                iterations=_iters(rng, 10, 200, nx, ny, 2e9))


# ----------------------------------------------------------------- inputs

def _noise(nx, ny, seed, base=4, octaves=8):
    """A fractal heightmap in [0, 1]: octaves of bicubically interpolated
    random lattices, halving in amplitude and doubling in frequency."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed & 0x7FFFFFFFFFFFFFFF)
    big = max(nx, ny)
    out = torch.zeros((ny, nx), device="cuda")
    for k in range(octaves):
        f = base * 2 ** k
        ly, lx = max(4, math.ceil(f * ny / big) + 3), max(4, math.ceil(f * nx / big) + 3)
        lat = torch.rand((1, 1, ly, lx), device="cuda", generator=g)
        if lx > 2 * nx or ly > 2 * ny:
            break
        out += 0.5 ** k * torch.nn.functional.interpolate(lat, size=(ny, nx), mode="bicubic", align_corners=False)[0, 0]
    out -= out.min()
    return (out / out.max()).contiguous()


def _grids(case, seed):
    """Named input grids of a case on the device, from the seed alone."""
    nx, ny, kind = case["nx"], case["ny"], case["kind"]
    seed = 1000003 * seed + 17
    big = max(nx, ny)
    g = {"z": _noise(nx, ny, seed)}
    if kind in ("deposition", "stencil") or (kind == "thermal" and case["talus"] == "map"):
        g["talus"] = (0.5 + _noise(nx, ny, seed + 1)) / big
    if kind == "thermal" and case["bedrock"]:
        g["bedrock"] = 0.3 * g["z"]
    if kind == "thermal" and case["mask"]:
        g["mask"] = _noise(nx, ny, seed + 2, octaves=3)
    if kind == "vpipes" and case["rain_map"]:
        g["rain"] = 0.25 + _noise(nx, ny, seed + 3, octaves=4)
    if kind in ("flow", "viscous"):
        g["depth"] = _noise(nx, ny, seed + 4, octaves=3)
    if kind == "viscous":
        # a smooth terrain: the film is stable on slopes of a few cells
        g["z"] = _noise(nx, ny, seed, octaves=3)
    if kind == "stencil" and case["rule"] == "scree":
        g["zmax"] = g["z"] + 0.25
    return g


def _talus_value(case):
    return float(np.float32(1.0 / max(case["nx"], case["ny"])))


def _specs(case):
    """Jobs of a batch: sides log-uniform, multiples of 8, aspect up to 2,
    thermal and vpipes in turn, uneven iterations."""
    rng = np.random.default_rng(case["jobseed"])
    out = []
    for k in range(case["jobs"]):
        a = math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"])))
        b = a / rng.uniform(1.0, 2.0)
        if rng.uniform() < 0.5:
            a, b = b, a
        nx, ny = (int(min(case["hi"], max(case["lo"], round(s / 8) * 8))) for s in (a, b))
        it = int(rng.integers(max(10, case["iterations"] // 4), case["iterations"] + 1))
        talus = float(np.float32(rng.uniform(0.5, 2.0) / nx))
        rain = float(np.float32(rng.uniform(5e-5, 5e-4)))
        out.append(dict(kind="thermal" if k % 2 == 0 else "vpipes", nx=nx, ny=ny, iterations=it, talus=talus,
                        rain=rain))
    return out


def prepare(case, seed):
    st = {"case": case}
    if case["kind"] == "batch":
        st["z0"] = [_noise(s["nx"], s["ny"], 7919 * seed + k) for k, s in enumerate(_specs(case))]
        st["z"] = [z.clone() for z in st["z0"]]
        st["jobs"] = [B.thermal_job(z, s["talus"], s["iterations"]) if s["kind"] == "thermal" else
                      B.vpipes_job(z, s["iterations"], **dict(RAIN, rain_per_step=s["rain"]))
                      for s, z in zip(_specs(case), st["z"])]
        torch.cuda.synchronize()
        return st
    g = _grids(case, seed)
    if case.get("host"):
        g = {k: v.cpu().numpy() for k, v in g.items()}
        empty = np.empty_like
    else:
        empty = torch.empty_like
    st.update(g)
    st["z0"] = st["z"]
    st["z"] = empty(st["z0"])
    if case["kind"] == "thermal":
        st["dep"] = empty(st["z0"]) if case["deposition"] else None
    elif case["kind"] == "vpipes":
        st["out"] = [empty(st["z0"]) if case["outputs"] else None for _ in range(4)]
        st["params"] = dict(RAIN if case["preset"] == "rain" else DEFAULTS, iterations=case["iterations"])
        if not case["host"]:
            st["params"] = G.vpipes_params(**st["params"])
    elif case["kind"] in ("flow", "viscous", "deposition") or case["rule"] in ("ridge", "scree"):
        st["out"] = empty(st["z0"])
    torch.cuda.synchronize()
    return st


# -------------------------------------------------------------------- run

def run(st):
    case = st["case"]
    kind = case["kind"]
    z, z0 = st["z"], st["z0"]
    if kind == "batch":
        for a, b in zip(z, z0):
            a.copy_(b)
        # the batch runs on its own streams: its inputs have to be there
        torch.cuda.current_stream().synchronize()
        B.run(st["jobs"])
        return z
    it = case.get("iterations")
    if case.get("host"):
        np.copyto(z, z0)
    elif kind in ("thermal", "vpipes", "deposition", "stencil"):
        z.copy_(z0)
    if kind == "thermal":
        talus = st["talus"] if case["talus"] == "map" else _talus_value(case)
        dep, mask = st["dep"], st.get("mask")
        if case["auto"]:
            f = G.thermal_auto_bedrock if case["host"] else G.thermal_auto_bedrock_device
            f(z, talus, it, deposition_map=dep, mask=mask)
        else:
            f = G.thermal if case["host"] else G.thermal_device
            f(z, talus, it, bedrock=st.get("bedrock"), deposition_map=dep, mask=mask)
        return [z] if dep is None else [z, dep]
    if kind == "vpipes":
        d, s, u, v = st["out"]
        if case["host"]:
            G.hydraulic_vpipes(z, rain_map=st.get("rain"), water_depth=d, sediment=s, vel_u=u, vel_v=v, **st["params"])
        else:
            G.hydraulic_vpipes_device(z, st["params"], rain_map=st.get("rain"), water_depth=d, sediment=s, vel_u=u,
                                      vel_v=v)
        return [z] + [a for a in st["out"] if a is not None]
    if kind == "flow":
        G.flow_simulation_device(z0, 0.01, st["depth"], it, st["out"], dry_out_ratio=case["dry_out"])
        return [st["out"]]
    if kind == "viscous":
        G.flow_simulation_viscous_device(z0, 0.01, st["depth"], it, st["out"], power=case["power"])
        return [st["out"]]
    if kind == "deposition":
        G.sediment_deposition_device(z, st["talus"], st["out"], 0.01, case["layers"], it)
        return [z, st["out"]]
    rule = case["rule"]
    if rule in ("ridge", "scree"):
        G.thermal_stencil_device(STENCILS[rule], z, st["talus"], it, zmax=st.get("zmax"), deposition_map=st["out"])
        return [z, st["out"]]
    G.thermal_relief_device(STENCILS[rule], z, st["talus"] if rule == "inflate" else None, it)
    return [z]


# ------------------------------------------------------------------- work

# arithmetic of one cell and step as the kernels' text has it (adds,
# multiplies, divisions, square roots and comparisons, each counted once)
_FLOPS = {"thermal": 60, "vpipes": 190, "flow": 65, "viscous": 40, "deposition": 60, "stencil": 60}


def work(case):
    kind = case["kind"]
    if kind == "batch":
        b = f = 0
        for s in _specs(case):
            n = s["nx"] * s["ny"]
            b += 8 * n
            f += _FLOPS[s["kind"]] * n * s["iterations"]
        return {"bytes": float(b), "flops": float(f)}
    n = case["nx"] * case["ny"]
    grids = 2  # the heights in and out
    if kind == "thermal":
        grids += sum((case["talus"] == "map", case["bedrock"], case["deposition"], case["mask"]))
    elif kind == "vpipes":
        grids += (1 if case["rain_map"] else 0) + (4 if case["outputs"] else 0)
    elif kind in ("flow", "viscous"):
        grids = 3
    elif kind == "deposition":
        grids += 2
    else:
        grids += {"ridge": 2, "scree": 3, "inflate": 1, "rib": 0}[case["rule"]]
    steps = case["iterations"] * case.get("layers", 1)
    return {"bytes": 4.0 * grids * n, "flops": float(_FLOPS[kind]) * n * steps}


# ------------------------------------------------------------------ exact

_DI = (-1, 0, 0, 1, -1, -1, 1, 1)
_DJ = (0, 1, -1, 0, -1, 1, -1, 1)


def _borders(a, b):
    """Border cells of b take their inward neighbour in a."""
    b[0, 1:-1] = a[1, 1:-1]
    b[-1, 1:-1] = a[-2, 1:-1]
    b[:, 0] = a[:, 1]
    b[:, -1] = a[:, -2]


def _extrapolate(a, nb=1):
    for k in range(nb - 1, -1, -1):
        a[:, k] = 2 * a[:, k + 1] - a[:, k + 2]
        a[:, -1 - k] = 2 * a[:, -2 - k] - a[:, -3 - k]
    for k in range(nb - 1, -1, -1):
        a[k] = 2 * a[k + 1] - a[k + 2]
        a[-1 - k] = 2 * a[-2 - k] - a[-3 - k]


def _around(a):
    """The eight neighbours of the interior cells, with their distances."""
    ny, nx = a.shape
    for k in range(8):
        i, j = 1 + _DI[k], 1 + _DJ[k]
        yield a[j:ny - 2 + j, i:nx - 2 + i], (1.0 if k < 4 else 1.414)


def _thermal64(z0, talus, iterations, bedrock=None, auto=False):
    """The heights after the steps and the border extrapolation."""
    a = z0.clone()
    t = talus if isinstance(talus, float) else talus[1:-1, 1:-1]
    bed = None if bedrock is None else bedrock[1:-1, 1:-1]
    for it in range(iterations):
        c = a[1:-1, 1:-1]
        amount = torch.zeros_like(c)
        for q, dist in _around(a):
            n = q - c
            amount += torch.sign(n) * torch.clamp(n.abs() - dist * t, min=0) * (0.2 / dist)
        new = c + amount
        if bed is not None:
            new = torch.maximum(torch.where(c >= bed, new, c), bed)
        if auto:
            new = torch.maximum(new, z0[1:-1, 1:-1])
            if it > 0:
                new = torch.maximum(new, c)
        b = torch.empty_like(a)
        b[1:-1, 1:-1] = new
        _borders(a, b)
        a = b
    _extrapolate(a)
    return a


def _finish64(z0, a, deposition, mask, absolute=False):
    out = [a if mask is None else z0 * (1 - mask) + a * mask]
    if deposition:
        out.append((a - z0).abs() if absolute else torch.clamp(a - z0, min=0))
    return out


def _shift(a, di, dj):
    """a at (i + di, j + dj), clamped to the grid."""
    p = torch.nn.functional.pad(a[None, None], (1, 1, 1, 1), mode="replicate")[0, 0]
    ny, nx = a.shape
    return p[1 + dj:1 + dj + ny, 1 + di:1 + di + nx]


def _flow_water64(z, d, f, p):
    """New fluxes (left, right, j + 1, j - 1), depth and velocity."""
    h = z + d
    dt, ga = p["dt"], p["gravity"] * p["pipe_area"]
    n = [torch.clamp(f[k] + dt * ga * (h - _shift(h, *o)), min=0)
         for k, o in enumerate(((-1, 0), (1, 0), (0, 1), (0, -1)))]
    if p["flux_diffusion"]:
        c0 = p["flux_diffusion_strength"]
        add = c0 * (n[0] + n[1] + n[2] + n[3])
        n = [(1 - 4 * c0) * q + add for q in n]
    tot = n[0] + n[1] + n[2] + n[3]
    k = torch.where(tot > p["floor"], d / (tot * dt), torch.zeros_like(d)).clamp(0, 1)
    n = [q * k for q in n]
    fw, fe, fn, fs = _shift(n[1], -1, 0), _shift(n[0], 1, 0), _shift(n[2], 0, -1), _shift(n[3], 0, 1)
    d2 = torch.clamp(d + dt * (fw + fn + fe + fs - n[0] - n[1] - n[2] - n[3]), min=0)
    dm = torch.clamp(d2, min=0.001 * p["water_height"] / dt)
    u = 0.5 * (fw - n[0] + n[1] - fe) / dm
    v = 0.5 * (fn - n[3] + n[2] - fs) / dm
    return n, d2, u, v


def _mirror(x, n):
    return (x - 2 * n * torch.round(x / (2 * n))).abs()


def _sample(s, x, y):
    """Bilinear sample, texel centres at k + 0.5, mirrored repeat."""
    ny, nx = s.shape
    x, y = _mirror(x, nx) - 0.5, _mirror(y, ny) - 0.5
    fx, fy = torch.floor(x), torch.floor(y)
    a, b = x - fx, y - fy
    i0, j0 = fx.long().clamp(-1, nx - 1), fy.long().clamp(-1, ny - 1)
    i1, j1 = (i0 + 1).clamp(max=nx - 1), (j0 + 1).clamp(max=ny - 1)
    i0, j0 = i0.clamp(min=0), j0.clamp(min=0)
    return ((1 - a) * (1 - b) * s[j0, i0] + a * (1 - b) * s[j0, i1] + (1 - a) * b * s[j1, i0] + a * b * s[j1, i1])


def _single(p):
    """Parameters as the call takes them: 32-bit floats."""
    return {k: float(np.float32(v)) for k, v in p.items()}


def _vpipes64(z, rain, p, iterations):
    p = _single(dict(p, flux_diffusion_strength=0.01, ratio=10.0, floor=1e-5))
    ny, nx = z.shape
    rain = torch.ones_like(z) if rain is None else rain
    d = (p["water_height"] if p["initial_water"] < 0 else p["initial_water"]) * rain
    v0, r = d.sum(), rain.sum()
    s = torch.zeros_like(z)
    f = [torch.zeros_like(z) for _ in range(4)]
    u = v = s
    gx = torch.arange(nx, device=z.device, dtype=z.dtype)[None, :]
    gy = torch.arange(ny, device=z.device, dtype=z.dtype)[:, None]
    for _ in range(iterations):
        d = d + p["rain_per_step"] * rain
        f, d2, u, v = _flow_water64(z, d, f, p)
        dzx = 0.5 * (_shift(z, 1, 0) - _shift(z, -1, 0) + _shift(s, 1, 0) - _shift(s, -1, 0))
        dzy = 0.5 * (_shift(z, 0, 1) - _shift(z, 0, -1) + _shift(s, 0, 1) - _shift(s, 0, -1))
        dzn = torch.clamp(nx * torch.hypot(dzx, dzy), min=1e-3)
        salpha = torch.clamp(dzn / torch.sqrt(1 + dzn * dzn), min=0.01)
        capa = p["k_capacity"] * torch.clamp(d2 / p["water_height"], max=p["ratio"]) * torch.hypot(u, v) * salpha
        up = capa > s
        change = torch.where(up, p["k_erode"] * (capa - s), -p["k_depose"] * (s - capa))
        z = z - change
        s = _sample(s + change, gx - p["dt"] * u, gy - p["dt"] * v)
        d = d2 * (1 - p["dt"] * p["evap_rate"])
        if p["maintain_water_volume"]:
            d = d + (v0 - d.sum()) * rain / r
    return [z, d, s, u, v]


def _flow64(z, depth, it, dry_out):
    p = _single(dict(dt=0.5, gravity=1.0, pipe_area=1.0, flux_diffusion=1, flux_diffusion_strength=0.01, floor=1e-5,
                     water_height=0.01, dry=dry_out))
    d = p["water_height"] * depth
    f = [torch.zeros_like(z) for _ in range(4)]
    for _ in range(it):
        f, d, _u, _v = _flow_water64(z, d, f, p)
    return [torch.clamp(d - p["dry"] * d.max(), min=0) if dry_out else d]


def _viscous64(z, depth, it, power):
    power, viscosity = float(np.float32(power)), 1.0
    h = float(np.float32(0.01)) * depth
    dt = 0.5
    for k in range(it):
        if k % 10 == 0:
            dt = 0.2 / torch.clamp(h.max() ** power / viscosity, min=1e-6)
        surf = h + z
        out = torch.zeros_like(h)
        for o in ((1, 0), (-1, 0), (0, 1), (0, -1)):
            m = (0.5 * (h + _shift(h, *o))) ** power / viscosity
            out += m * (_shift(surf, *o) - surf)
        h = torch.clamp(h + dt * out, min=0)
    return [h]


def _deposition64(z, talus, layers, it):
    sed = torch.zeros_like(z)
    step = float(np.float32(0.01)) / layers
    for _ in range(layers):
        sed = torch.clamp(_thermal64(z + sed + step, talus, it) - z, min=0)
    return [z + sed, sed]


def _stencil64(rule, z0, talus, zmax, it):
    a = z0.clone()
    for _ in range(it):
        c = a[1:-1, 1:-1]
        total, steep = torch.zeros_like(c), torch.zeros_like(c)
        least = torch.full_like(c, math.inf)
        for q, dist in _around(a):
            dz = (c - q) / dist
            total += torch.clamp(dz, min=0) if rule == "ridge" else torch.clamp(dz, max=0)
            steep = torch.maximum(steep, dz.abs())
            least = torch.minimum(least, dz.abs())
        b = torch.empty_like(a)
        if rule == "rib":
            b[1:-1, 1:-1] = c - least
        else:
            t = talus[1:-1, 1:-1]
            amp = torch.clamp(1 - t / steep, 0, 1)
            amp = amp * amp * (3 - 2 * amp)
            if rule == "scree":
                x = torch.clamp(1 - c / zmax[1:-1, 1:-1], 0, 1)
                amp = amp * (2 - x) * x * x
            b[1:-1, 1:-1] = c + 0.25 * (t - 0.5 * total) * amp
        _borders(a, b)
        a = b
    _extrapolate(a, 3 if rule == "rib" else 1)
    return a


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        out = []
        for k, s in enumerate(_specs(case)):
            z = _noise(s["nx"], s["ny"], 7919 * seed + k).double()
            if s["kind"] == "thermal":
                out.append(_thermal64(z, s["talus"], s["iterations"]))
            else:
                out.append(_vpipes64(z, None, dict(RAIN, rain_per_step=s["rain"]), s["iterations"])[0])
        return out
    g = {k: v.double() for k, v in _grids(case, seed).items()}
    z = g["z"]
    if kind == "thermal":
        talus = g["talus"] if case["talus"] == "map" else _talus_value(case)
        a = _thermal64(z, talus, case["iterations"], g.get("bedrock"), case["auto"])
        out = _finish64(z, a, case["deposition"], g.get("mask"))
    elif kind == "vpipes":
        out = _vpipes64(z, g.get("rain"), RAIN if case["preset"] == "rain" else DEFAULTS, case["iterations"])
        out = out if case["outputs"] else out[:1]
    elif kind == "flow":
        out = _flow64(z, g["depth"], case["iterations"], case["dry_out"])
    elif kind == "viscous":
        out = _viscous64(z, g["depth"], case["iterations"], case["power"])
    elif kind == "deposition":
        out = _deposition64(z, g["talus"], case["layers"], case["iterations"])
    else:
        rule = case["rule"]
        a = _stencil64(rule, z, g.get("talus"), g.get("zmax"), case["iterations"])
        out = _finish64(z, a, rule in ("ridge", "scree"), None, absolute=rule == "ridge")
    return [a.cpu().numpy() for a in out] if case.get("host") else out
