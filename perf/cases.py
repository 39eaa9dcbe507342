"""Timed cases of the multiple-scattering path, through the Python interface
over the C ABI: what programs that use this package have it do.

A case is a dict of plain values; ``do`` says which call it times:

  solve     LightGraph over point clouds: graph build, edge march, all-pairs
            paths, vertex light and diffusion; the diffused radiances come back
  darts     LightGraph.scatterPoints: the point clouds of a range of iterations
  flow      LightGraph, ScatterGrid, VolumeRender one after the other, with
            every stage's result taken to the host
  frame     Context.render_frame: points in, four films out
  pipeline  the whole pipeline without injected points: dart throwing, solve,
            splat and render of a range of iterations
  render    VolumeRender.render of a solved scene (a new camera or more
            samples over the same scatter grid)
  sequence  a frame of an animated volume: the new grids go to the device,
            then render_frame
  paths     all-pairs shortest paths of a dense matrix on the host

The volumes are the seeded synthetic clouds of lightgraph_gb300.scenes; the
seed of a case moves the points, the lights, the camera and the random
streams.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from lightgraph_gb300 import Context, LightGraph, ScatterGrid, VolumeRender, _capi, scenes
from lightgraph_gb300.lightgraph import ColorRamp, Grid, Light, SceneSettings, Shader

DTYPES = {"f32": _capi.LG_DTYPE_F32, "f16": _capi.LG_DTYPE_F16, "bf16": _capi.LG_DTYPE_BF16}
SUN, LAMP, SKY = (1.0, 0.89, 0.79), (0.4, 0.6, 1.0), (1.0, 1.0, 1.0)


def listed():
    return [
        # an artist's preview solve: one small cloud, where latency and launches count
        {"name": "solve-preview", "do": "solve", "res": 64, "graphs": 1, "n_min": 200, "n_max": 200, "radius": 0.3,
         "lights": "sun", "dtype": "f32"},
        # clouds of the size that dart throwing makes (about 750 points), many iterations at once
        {"name": "solve-iterations", "do": "solve", "res": 256, "graphs": 48, "n_min": 737, "n_max": 751,
         "radius": 0.12, "lights": "sun+lamp", "dtype": "f32"},
        # the production scene's one 4096-point cloud
        {"name": "solve-production", "do": "solve", "res": 256, "graphs": 1, "n_min": 4096, "n_max": 4096,
         "radius": 0.075, "lights": "sun+lamp", "dtype": "f32"},
        # clouds of uneven size in one call, half-precision volume
        {"name": "solve-uneven", "do": "solve", "res": 256, "graphs": 32, "n_min": 257, "n_max": 3805, "radius": 0.15,
         "lights": "sun", "dtype": "f16"},
        # the point clouds of some iterations, 1M candidates each
        {"name": "darts", "do": "darts", "res": 256, "iterations": 48, "dtype": "f32"},
        # the three classes in a row on the small scene, as the README has it
        {"name": "flow-small", "do": "flow", "res": 128, "points": 1024, "radius": 0.15, "lights": "sun",
         "width": 256, "height": 256, "spp": 1, "dtype": "f32"},
        # the production frame: 512^3 cumulus with temperature, two lights, 1024^2 at 4 spp
        {"name": "frame-production", "do": "frame", "res": 512, "points": 4096, "radius": 0.075, "lights": "sun+lamp",
         "width": 1024, "height": 1024, "spp": 4, "dtype": "f32", "fire": True},
        # the reference's own scene shape with fewer iterations: darts, sun and a 3-sample sky, 960x540 at 3 spp
        {"name": "pipeline-sky", "do": "pipeline", "res": 512, "iterations": 24, "lights": "sun+sky3", "width": 960,
         "height": 540, "spp": 3, "dtype": "f32", "fire": True},
        # look development under a sky: an odd image over a half-precision volume
        {"name": "render-sky-half", "do": "render", "res": 208, "points": 1500, "radius": 0.11, "lights": "sun+sky2",
         "width": 411, "height": 307, "spp": 2, "dtype": "f16", "fire": False},
        # a thumbnail with a lamp: the smallest render
        {"name": "render-thumbnail", "do": "render", "res": 96, "points": 300, "radius": 0.2, "lights": "lamp",
         "width": 121, "height": 89, "spp": 1, "dtype": "bf16", "fire": False},
        # an animation: new grids every frame
        {"name": "sequence", "do": "sequence", "res": 192, "points": 700, "radius": 0.13, "lights": "sun+lamp",
         "width": 480, "height": 270, "spp": 1, "dtype": "f32", "fire": True},
        # a dense matrix of any origin, directed edges, odd size
        {"name": "paths-dense", "do": "paths", "n": 1021, "density": 0.02},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _res(rng, lo, hi):
    return max(lo, min(hi, 16 * round(_log(rng, lo, hi) / 16)))  # brick-aligned origin


def draw(rng):
    do = rng.choice(["solve", "solve", "solve", "darts", "flow", "frame", "frame", "pipeline", "render", "render",
                     "sequence", "paths"])
    dtype = rng.choice(["f32", "f32", "f16", "bf16"])
    if do == "paths":
        return {"do": do, "n": _log(rng, 60, 2100), "density": round(rng.uniform(0.01, 0.05), 3)}
    if do == "darts":
        return {"do": do, "res": _res(rng, 64, 256), "iterations": _log(rng, 4, 64), "dtype": dtype}
    if do == "solve":
        graphs = _log(rng, 1, 48)
        top = _log(rng, 65, 4096 if graphs < 32 else 2048)
        low = top if rng.random() < 0.4 else _log(rng, 33, top)
        # about 20 neighbours inside the radius, as the listed clouds have
        return {"do": do, "res": _res(rng, 64, 256), "graphs": graphs, "n_min": low, "n_max": top,
                "radius": round(1.15 * top ** (-1.0 / 3.0), 3), "lights": rng.choice(["sun", "lamp", "sun+lamp"]),
                "dtype": dtype}
    small = {"width": _log(rng, 60, 640), "height": _log(rng, 40, 480), "spp": rng.choice([1, 1, 2, 3, 4]),
             "dtype": dtype}
    lights = rng.choice(["sun", "lamp", "sun+lamp", "sun+sky1", "sky2", "sun+sky3"])
    if do == "pipeline":
        return dict({"do": do, "res": _res(rng, 96, 256), "iterations": _log(rng, 3, 24), "lights": lights,
                     "fire": rng.random() < 0.5}, **small)
    n = _log(rng, 100, 2500)
    case = dict({"do": do, "res": _res(rng, 64, 256), "points": n, "radius": round(1.15 * n ** (-1.0 / 3.0), 3),
                 "lights": lights}, **small)
    if do != "flow":
        case["fire"] = rng.random() < 0.5
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _density(res):
    return scenes.volume(_capi.LGS_VOLUME_CUMULUS, res, 6, 1)


@functools.lru_cache(maxsize=None)
def _temperature(res):
    return scenes.volume(_capi.LGS_VOLUME_TEMPERATURE, res, 6, 2, 1500.0, mask=_density(res))


@functools.lru_cache(maxsize=None)
def _sky():
    return scenes.envmap()


def _grid(values, res):
    return Grid(values, (-res // 2,) * 3, 1.28 / res)


def _shader(res, fire):
    sh = Shader()
    k = 20.0 * 1.28 / res  # extinction 20 per world unit
    sh.setScattering((0.9 * k, 0.9 * k * 1.1, 0.9 * k * 1.25))
    sh.setAbsorption(0.1 * k)
    sh.setScatterScale(4.0 * 0.9 * k / 1.5)
    if fire:
        sh.setEmissionScale(0.5)
        sh.setEmissionColorRamp(ColorRamp.parse(
            "0.0,0.33,0.66,1.0/0,0,0:1.0,0.076,0.0:1.0,0.322,0.0:1.0,0.45,0.15/600/1500"))
    return sh


def _lights(spec, rng):
    """The lights of a case: a sun, a lamp near the cloud, a sky of some samples."""
    out, sky = [], None
    for word in spec.split("+"):
        if word == "sun":
            turn = rng.uniform(20.0, 60.0)
            out.append(Light.parse("dir:0:%g,%g,%g:1.2:-40,%.3f,0" % (*SUN, turn)))
        elif word == "lamp":
            x = rng.uniform(0.5, 0.7)
            out.append(Light.parse("point:0:%g,%g,%g:30:%.3f,0.5,0.9" % (*LAMP, x)))
        else:
            sky = _sky()
            out.append(Light.parse("env:%.3f:%g,%g,%g:0.35:%s:sky" % (rng.uniform(0, 90), *SKY, word[3:])))
    return out, sky


def _settings(case, seed, rng):
    return SceneSettings(width=case.get("width", 64), height=case.get("height", 64), samples=case.get("spp", 1),
                         camTranslate=(0.0, 0.0, 2.2), camYRotate=float(rng.uniform(-20.0, 20.0)),
                         iter=case.get("iterations", case.get("graphs", 1)), seed=int(seed) & 0x7FFFFFFF)


def _context(case, seed, rng):
    res = case["res"]
    ctx = Context(0)
    ctx.upload_density(_grid(_density(res), res), DTYPES[case["dtype"]])
    if case.get("fire"):
        ctx.upload_temperature(_grid(_temperature(res), res), DTYPES[case["dtype"]])
    ctx.set_shader(_shader(res, case.get("fire")))
    opts = _settings(case, seed, rng)
    ctx.set_settings(opts)
    lights, sky = _lights(case.get("lights", "sun"), rng)
    ctx.set_lights(lights, sky)
    return ctx, opts, lights


def _sizes(case):
    """Cloud sizes, log-uniform between n_min and n_max; the same for every seed."""
    u = np.random.default_rng(case["graphs"]).random(case["graphs"])
    lo, hi = math.log(case["n_min"]), math.log(case["n_max"] + 0.99)
    return [int(math.exp(lo + (hi - lo) * x)) for x in u]


def _clouds(case, seed):
    """The point clouds of a solve."""
    res = case["res"]
    return [scenes.points(_density(res), 1.28 / res, int(n), int(seed % 100003) * 101 + g)
            for g, n in enumerate(_sizes(case))]


def _matrix(case, rng):
    """Random directed edges, with a ring so that every vertex can be reached."""
    n = case["n"]
    m = rng.random((n, n), dtype=np.float32) * 3.0 + 0.01
    m[rng.random((n, n), dtype=np.float32) > case["density"]] = np.inf
    at = np.arange(n)
    m[at, (at + 1) % n] = rng.random(n, dtype=np.float32) + 0.01
    np.fill_diagonal(m, 0.0)
    return m


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    do = case["do"]
    if do == "paths":
        return {"case": case, "ctx": Context(0), "matrix": _matrix(case, rng)}
    ctx, opts, lights = _context(case, seed, rng)
    state = {"case": case, "ctx": ctx, "opts": opts, "lights": lights}
    if do == "solve":
        state["clouds"] = _clouds(case, seed)
        state["radius"] = [case["radius"]] * case["graphs"]
    elif do in ("flow", "frame", "render", "sequence"):
        state["clouds"] = _clouds(dict(case, graphs=1, n_min=case["points"], n_max=case["points"]), seed)
        state["radius"] = [case["radius"]]
        state["radius_sq"] = [np.float32(case["radius"]) * np.float32(case["radius"])]
    if do == "render":
        LightGraph(ctx)(state["clouds"], state["radius"])
        ctx.splat()
    if do == "sequence":
        res, fire = case["res"], case.get("fire")
        scale = np.float32(rng.uniform(0.8, 1.0))  # this frame's volume
        state["density"] = _grid(_density(res) * scale, res)
        state["temperature"] = _grid(_temperature(res) * scale, res) if fire else None
    if do in ("darts", "pipeline"):
        state["first"] = int(seed) % 10000
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def _padded(rows, limit):
    """Per-iteration results of varying length as one array (1000 points an iteration at most)."""
    out = np.zeros((len(rows), limit, 3), np.float32)
    for k, r in enumerate(rows):
        out[k, :len(r)] = r
    return out


def _films(f):
    return {"rgba": f.rgba, "direct": f.direct, "scatter": f.scatter, "emission": f.emission}


def run(state):
    case, ctx = state["case"], state["ctx"]
    do = case["do"]
    if do == "paths":
        return ctx.fw_host(state["matrix"])
    if do == "solve":
        return LightGraph(ctx)(state["clouds"], state["radius"])
    if do == "darts":
        points, radius = LightGraph(ctx).scatterPoints(state["first"], case["iterations"])
        return {"points": _padded(points, 1000), "counts": np.array([len(p) for p in points]),
                "radius": np.array(radius)}
    if do == "flow":
        radiance = LightGraph(ctx)(state["clouds"], state["radius"])
        lo, dims, values = ScatterGrid(ctx)()
        films = VolumeRender(ctx, state["opts"]).render()
        return {"radiance": radiance, "lo": lo, "dims": dims, "grid": values, "films": _films(films)}
    if do == "frame":
        return _films(ctx.render_frame(state["clouds"], state["radius_sq"], state["opts"]))
    if do == "pipeline":
        counts = ctx.scatter_graphs(state["first"], case["iterations"])
        radiance = ctx.solve_graphs(want=True)
        ctx.splat()
        return dict(_films(ctx.render(state["opts"])), counts=counts,
                    radiance=_padded(np.split(radiance, np.cumsum(counts)[:-1]), 1000))
    if do == "render":
        return _films(VolumeRender(ctx, state["opts"]).render())
    if do == "sequence":
        dtype = DTYPES[case["dtype"]]
        ctx.upload_density(state["density"], dtype)
        if state["temperature"] is not None:
            ctx.upload_temperature(state["temperature"], dtype)
        return _films(ctx.render_frame(state["clouds"], state["radius_sq"], state["opts"]))
    raise ValueError(do)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def _solve_work(sizes):
    """Points in, radiances out; a relaxation per source and directed edge (at
    most 12 a vertex: an add and a minimum), and per pair the three
    transmittances, their column sums and the products of the diffusion."""
    pairs = float(sum(int(n) ** 2 for n in sizes))
    return 24.0 * float(sum(sizes)), pairs * (2 * 12 + 12)


def _render_work(case):
    """Film writes and one read of the cloud's voxels; per pixel sample about
    19 shading samples at 512^3 with one shadow ray per light sample, each ray
    about 21 density samples of about 20 operations (a trilinear sample, the
    step and the sum), in proportion to the resolution."""
    k = case["res"] / 512.0
    rays = 0
    for word in case["lights"].split("+"):
        rays += int(word[3:]) if word.startswith("sky") else 1
    samples = float(case["width"] * case["height"] * case["spp"])
    voxels = 0.14 * case["res"] ** 3 * (4 if case["dtype"] == "f32" else 2) * (2 if case.get("fire") else 1)
    return 64.0 * case["width"] * case["height"] + voxels, samples * (60 * k * 30 + 19 * k * rays * 21 * k * 20)


def work(case):
    do = case["do"]
    if do == "paths":
        return {"bytes": 8.0 * case["n"] ** 2, "flops": 2.0 * case["n"] ** 3}
    if do == "solve":
        b, f = _solve_work(_sizes(case))
        return {"bytes": b, "flops": f}
    if do == "darts":
        # 1M candidates an iteration: three draws, a position and a density sample each
        return {"bytes": 9000.0 * case["iterations"], "flops": 50e6 * case["iterations"]}
    b, f = _render_work(case)
    if do == "pipeline":
        sb, sf = _solve_work([750] * case["iterations"])
        return {"bytes": b + sb, "flops": f + sf + 50e6 * case["iterations"]}
    if do != "render":
        sb, sf = _solve_work([case["points"]])
        b, f = b + sb, f + sf
    if do == "flow":
        b += 12.0 * (case["res"] / 4) ** 3
    if do == "sequence":
        b += 4.0 * case["res"] ** 3 * (2 if case.get("fire") else 1)
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------

def _paths64(m):
    """Floyd-Warshall, a round at a time."""
    for k in range(m.shape[0]):
        torch.minimum(m, m[:, k:k + 1] + m[k:k + 1, :], out=m)
    return m


def _edges64(points, r2, cap):
    """buildGraph: rows in order, partners j > i inside the radius in order, while neither end is full."""
    n = len(points)
    count = np.zeros(n, np.int64)
    edges = []
    for i in range(n - 1):
        need = cap - count[i]
        if need <= 0:
            continue
        d = points[i] - points[i + 1:]
        near = np.flatnonzero(d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2] < r2) + i + 1
        near = near[count[near] < cap][:need]
        count[near] += 1
        edges.append(np.stack([np.full(len(near), i), near], 1))
    return np.concatenate(edges) if edges else np.zeros((0, 2), np.int64)


def _march64(vol, leaf, res, start, step_dir, length, step, take):
    """Sums take(density) * step at the multiples of step along the rays, where a leaf exists."""
    tau = torch.zeros(len(start), dtype=torch.float64, device=vol.device)
    top = float(length.max()) if len(length) else 0.0
    for k in range(1, int(min(top, 2.0 * res) // step) + 1):
        t = k * step
        on = torch.nonzero(length >= t).flatten()
        p = start[on] + t * step_dir[on] + res // 2
        c = torch.floor(p).long()
        inside = ((c >= 0) & (c < res)).all(1)
        on, p, c = on[inside], p[inside], c[inside]
        b = c // 8
        has = leaf[b[:, 2], b[:, 1], b[:, 0]]
        on, p, c = on[has], p[has], c[has]
        w = p - c
        rho = torch.zeros(len(on), dtype=torch.float64, device=vol.device)
        for corner in range(8):
            o = torch.tensor([corner & 1, corner >> 1 & 1, corner >> 2], device=vol.device)
            q = c + o
            f = torch.where(o.bool(), w, 1.0 - w).prod(1)
            ok = (q < res).all(1)
            q = q.clamp(max=res - 1)
            rho += torch.where(ok, vol[q[:, 2], q[:, 1], q[:, 0]].double(), 0.0) * f
        tau[on] += take(rho) * step
    return tau


def _solve64(case, seed):
    """The solve of every cloud in 64 bits (distant and point lights)."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    rng = np.random.default_rng(seed)
    res, voxel = case["res"], 1.28 / case["res"]
    rng_settings = _settings(case, seed, rng)
    lights, _ = _lights(case["lights"], rng)
    clouds = _clouds(case, seed)
    sh = _shader(res, False)
    host = torch.from_numpy(_density(res)).to(dev)
    vol = host.to({"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}[case["dtype"]])
    nb = res // 8
    leaf = (host.view(nb, 8, nb, 8, nb, 8) != 0).any(5).any(3).any(1)
    ext = torch.tensor([-e for e in sh.getExtinction()], dtype=torch.float64, device=dev)
    albedo = torch.tensor(sh.getAlbedo(), dtype=torch.float64, device=dev)
    scale = sh.density_scale * sh.shadow_density_scale * sh.scatter_density_scale
    cutoff, step = rng_settings.cutoff, rng_settings.step[1]
    dropped = lambda tau: torch.exp(-2.0 * tau[:, None] * ext).sum(1) < cutoff  # noqa: E731
    dens = lambda rho: (rho * scale).clamp(max=sh.density_max)  # noqa: E731
    lit = lambda rho: torch.where(dens(rho) < cutoff, 0.0, dens(rho))  # noqa: E731
    out = []
    for cloud, radius in zip(clouds, [case["radius"]] * case["graphs"]):
        n = len(cloud)
        e = torch.from_numpy(_edges64(cloud.astype(np.float64), float(np.float32(radius) * np.float32(radius)), 12))
        e = e.to(dev)
        p = torch.from_numpy(cloud).to(dev).double()
        d = p[e[:, 1]] - p[e[:, 0]]
        length = d.norm(dim=1)
        tau = _march64(vol, leaf, res, p[e[:, 0]] / voxel, d / length[:, None], length / voxel, step,
                       lambda rho: dens(rho).clamp(min=sh.scatter_density_min))
        tau = torch.where(dropped(tau), math.inf, tau)
        m = torch.full((n, n), math.inf, dtype=torch.float64, device=dev)
        m[e[:, 0], e[:, 1]] = tau
        m[e[:, 1], e[:, 0]] = tau
        m.fill_diagonal_(0.0)
        m = _paths64(m)
        light = torch.zeros((n, 3), dtype=torch.float64, device=dev)
        for lt in lights:
            power = torch.tensor([c * lt.c.intensity for c in lt.c.color], dtype=torch.float64, device=dev)
            if lt.type == _capi.LG_LIGHT_POINT:
                to = torch.tensor(list(lt.c.pos), dtype=torch.float64, device=dev) - p
                far = to.norm(dim=1)
                way, power = to / far[:, None], power / (1.0 + 4.0 * math.pi * far * far)[:, None]
                far = far / voxel
            else:
                way = -torch.tensor(list(lt.c.dir), dtype=torch.float64, device=dev).expand(n, 3)
                far = torch.full((n,), math.inf, dtype=torch.float64, device=dev)
            tau = _march64(vol, leaf, res, p / voxel, way, far, step, lit)
            seen = torch.where(dropped(tau), 0.0, 1.0)[:, None]
            light += albedo * power * torch.exp(-tau[:, None] * ext) * seen
        got = torch.empty((n, 3), dtype=torch.float64, device=dev)
        for c in range(3):
            t = torch.exp(-ext[c] * m)
            got[:, c] = t @ (light[:, c] / t.sum(0).clamp(min=1.0))
        out.append(got.cpu().numpy())
    return out


def exact(case, seed):
    if case["do"] == "paths":
        m = torch.from_numpy(_matrix(case, np.random.default_rng(seed))).double()
        return _paths64(m.cuda() if torch.cuda.is_available() else m).cpu().numpy()
    if case["do"] == "solve":
        return _solve64(case, seed)
    # the dart sequence takes minutes in plain code; an image is a Monte Carlo
    # estimate over this package's own random streams and has no other value
    return None
