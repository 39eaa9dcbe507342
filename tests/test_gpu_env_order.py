"""Environment-light shadow rays in sorted order (more than four million rays
through a box whose records exceed the L2, EnvOrder): image rows against the
FP64 oracle, which marches them ray by ray. Each AOV's relative RMSE <= 1e-3,
as for every frame compared with the oracle."""
import numpy as np
import pytest

from lightgraph_gb300 import scenes
from lightgraph_gb300.lightgraph import Grid, Light, SceneSettings, Shader
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


def rel_rmse(a, b):
    a, b = a.astype(np.float64), b.astype(np.float64)
    den = np.sqrt(np.mean(b * b))
    return float(np.sqrt(np.mean((a - b) ** 2)) / (den if den else 1.0))


@pytest.mark.parametrize("dtype, samples", [(0, 2), (1, 1)])
def test_sorted_rays_match_oracle(gpu_ctx, dtype, samples):
    n, depth, h = 520, 72, 0.0025
    z, y, x = np.meshgrid(np.arange(depth), np.arange(n), np.arange(n), indexing="ij", sparse=True)
    v = (0.25 + 0.2 * np.sin(x * 0.11) * np.cos(y * 0.07) + 0.1 * np.sin(z * 0.3 + x * 0.02)).astype(np.float32)
    if dtype == 1:
        v = v.astype(np.float16).astype(np.float32)
    grid = Grid(np.ascontiguousarray(v), (-264, -264, -40), h)
    sh = Shader()
    k = 20.0 * h
    sh.setScattering((0.9 * k, 0.95 * k, 1.0 * k))
    sh.setAbsorption(0.1 * k)
    opts = SceneSettings(width=640, height=480, samples=1, camTranslate=(0.0, 0.0, 1.4), iter=1, seed=3)
    lights = [Light.parse("dir:0:1,0.9,0.8:1.0:-35,25,0"), Light.parse(f"env:20:1,1,1:0.5:{samples}:sky")]
    sky = scenes.envmap(64, 32)
    gpu_ctx.upload_density(grid, dtype)
    gpu_ctx.upload_temperature(None)
    gpu_ctx.set_shader(sh)
    gpu_ctx.set_settings(opts)
    gpu_ctx.set_lights(lights, sky)
    pts = [scenes.points(np.full((64, 64, 64), 0.5, np.float32), 0.002, 64, 5)]
    gpu_ctx.build_graphs(pts, [np.float32(0.05) ** 2], 12)
    gpu_ctx.solve_graphs()
    gpu_ctx.splat()
    films = gpu_ctx.render(opts)
    assert gpu_ctx.shading_tasks() >= 4 << 20
    lo, dims, vals = gpu_ctx.scatter_grid()
    o = po.Oracle(grid, sh, opts, lights, env_map=sky)
    rows = [60, 241, 402]
    ref = o.render((lo, dims, vals), rows=rows)
    for i, name in enumerate(("rgba", "direct", "scatter", "emission")):
        assert rel_rmse(getattr(films, name)[rows], ref[i][rows]) <= 1e-3, name


def test_small_frames_after_a_large_one(gpu_ctx):
    """Whether a frame's rays are sorted is decided by that frame: after a large
    one a thumbnail over the same volume takes the launches and gives the bits
    that it does on a context of its own, captured or not."""
    from lightgraph_gb300 import Context
    n, depth, h = 520, 72, 0.0025
    v = np.full((depth, n, n), 0.3, np.float32)
    grid = Grid(v, (-264, -264, -40), h)
    sh = Shader()
    sh.setScattering((0.05, 0.05, 0.05))
    sh.setAbsorption(0.005)
    lights = [Light.parse("dir:0:1,0.9,0.8:1.0:-35,25,0"), Light.parse("env:20:1,1,1:0.5:2:sky")]
    sky = scenes.envmap(64, 32)
    pts = [scenes.points(np.full((64, 64, 64), 0.5, np.float32), 0.002, 64, 5)]
    r2 = [np.float32(0.05) ** 2]

    def settings(w, hgt):
        return SceneSettings(width=w, height=hgt, samples=1, camTranslate=(0.0, 0.0, 1.4), iter=1, seed=3)

    def load(ctx):
        ctx.upload_density(grid)
        ctx.upload_temperature(None)
        ctx.set_shader(sh)
        ctx.set_settings(settings(48, 32))
        ctx.set_lights(lights, sky)
        ctx.build_graphs(pts, r2, 12)
        ctx.solve_graphs()
        ctx.splat()

    def thumbnail(ctx):
        before = ctx.kernel_launches()
        films = ctx.render(settings(48, 32))
        launches = ctx.kernel_launches() - before
        ctx.set_graph_mode(True)
        ctx.frame_device(settings(48, 32))
        captured = int(ctx.lib.lg_frame_launches(ctx.h))
        ctx.frame_device(settings(48, 32))
        replayed = ctx.films(settings(48, 32))
        ctx.set_graph_mode(False)
        return films, replayed, launches, captured

    other = Context(0)
    load(other)
    films, replayed, launches, captured = thumbnail(other)
    other.close()
    load(gpu_ctx)
    before = gpu_ctx.kernel_launches()
    gpu_ctx.render(settings(640, 480))
    assert gpu_ctx.shading_tasks() >= 4 << 20
    assert gpu_ctx.kernel_launches() - before > launches  # sorted
    got = thumbnail(gpu_ctx)
    assert got[2:] == (launches, captured)
    for name in ("rgba", "direct", "scatter", "emission"):
        assert np.array_equal(getattr(got[0], name), getattr(films, name)), name
        assert np.array_equal(getattr(got[1], name), getattr(replayed, name)), name
