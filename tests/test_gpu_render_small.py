"""Images of so few pixel samples that the shading pass fetches each sample's
density record ahead of the one before (k_primary), and one just past that size:
rows against the FP64 oracle over the same scatter grid, relative RMSE <= 1e-3 as
for every image compared with the oracle; the storage types read values that
they hold exactly."""
import numpy as np
import pytest

from lightgraph_gb300 import scenes
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


def rel_rmse(a, b):
    a, b = a.astype(np.float64), b.astype(np.float64)
    den = np.sqrt(np.mean(b * b))
    return float(np.sqrt(np.mean((a - b) ** 2)) / (den if den else 1.0))


def held(v, dtype):
    if dtype == 1:
        v = v.astype(np.float16).astype(np.float32)
    elif dtype == 2:
        v = (v.view(np.uint32) & np.uint32(0xFFFF0000)).view(np.float32)
    return np.ascontiguousarray(v)


@pytest.mark.parametrize("dtype", [0, 1, 2])
@pytest.mark.parametrize("width, height, spp", [(1, 1, 1), (7, 3, 2), (33, 20, 1), (432, 360, 1), (433, 360, 1)])
def test_rows_match_oracle(gpu_ctx, width, height, spp, dtype):
    sc = scenes.production(n_points=64, width=width, height=height, spp=spp, res=64)
    sc.density.values = held(sc.density.values, dtype)
    sc.temperature.values = held(sc.temperature.values, dtype)
    scenes.load_into(gpu_ctx, sc, dtype)
    gpu_ctx.build_graphs(sc.points, sc.radius_sq, sc.max_connect)
    gpu_ctx.solve_graphs()
    gpu_ctx.splat()
    films = gpu_ctx.render(sc.opts)
    again = gpu_ctx.render(sc.opts)
    grid = gpu_ctx.scatter_grid()
    o = po.Oracle(sc.density, sc.shader, sc.opts, sc.lights, temperature=sc.temperature)
    rows = list(range(height)) if height <= 20 else [90, 181, 240]
    ref = o.render(grid, rows=rows)
    for i, name in enumerate(("rgba", "direct", "scatter", "emission")):
        film = getattr(films, name)
        assert np.array_equal(film, getattr(again, name))
        assert rel_rmse(film[rows], ref[i][rows]) <= 1e-3, name
