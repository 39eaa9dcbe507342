"""The path solve from the edges (k_paths.cu), which runs where no Floyd-Warshall
schedule is pinned and the graphs are few or large: graph sizes around a source group, a mark
word and the sizes at which the group or the thread count changes, edge caps
off the usual 12, graphs in several pieces and empty ones, batches of mixed
sizes. The diffused radiances against the oracle's (FP64 Dijkstra over the
GPU's own edge depths, then its diffusion) and against the pinned
Floyd-Warshall solve, 1e-4 relative as elsewhere; two runs give the same
bits."""
import numpy as np
import pytest

from lightgraph_gb300 import scenes
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene():
    return scenes.small(n_points=16, width=16, height=16, res=64)


def solve(ctx, sc, clouds, radius, cap, oracle=True):
    scenes.load_into(ctx, sc)
    ctx.set_fw_schedule(-1)
    r2 = [np.float32(r) * np.float32(r) for r in radius]
    ctx.build_graphs(clouds, r2, cap)
    D = ctx.solve_graphs(want=True)
    assert np.array_equal(D, ctx.solve_graphs(want=True))
    L, _ = ctx.vertex_data()
    S = ctx.march_edges(want=True)
    ctx.set_fw_schedule(4)
    fw = ctx.solve_graphs(want=True)
    ctx.set_fw_schedule(-1)
    assert np.allclose(D, fw, rtol=1e-4, atol=1e-7)
    L = L.astype(np.float64)
    if oracle:
        o = po.Oracle(sc.density, sc.shader, sc.opts, sc.lights)
        at = 0
        for s, c in zip(S, clouds):
            n = len(c)
            if n > 0:
                ref = o.diffuse(po.transmittance_of(po.apsp_dijkstra_f64(s), sc.shader.getExtinction()), L[at:at + n])
                assert np.allclose(D[at:at + n], ref, rtol=1e-4, atol=1e-7), n
            at += n


def cloud(sc, n, seed):
    if n == 0:
        return np.zeros((0, 3), np.float32)
    return scenes.points(sc.density.values, sc.density.voxel_size, n, seed)


@pytest.mark.parametrize("cap", [1, 2, 5, 12, 15, 16, 17])
def test_sizes(gpu_ctx, scene, cap):
    sizes = [0, 1, 2, 3, 4, 5, 15, 16, 17, 31, 33, 64, 65, 129, 500]
    clouds = [cloud(scene, n, 40 + n) for n in sizes]
    # a sparse radius leaves many pieces; 17 is past the cap the edges are used
    # for; the small graphs go by their edges alone or next to a large one
    for c in clouds:
        solve(gpu_ctx, scene, [c], [0.12], cap)
    solve(gpu_ctx, scene, clouds + [cloud(scene, 2049, 3)], [0.12] * (len(sizes) + 1), cap)


@pytest.mark.parametrize("sizes", [[1700, 1701, 2049, 300], [3040, 3041, 17], [1672], [1673], [2432], [2433], [700] * 5, [512] * 8, [300] * 9, [2300] + [400] * 16, [2300] + [900] * 16, [820] * 5])
def test_group_sizes(gpu_ctx, scene, sizes):
    clouds = [cloud(scene, n, 7 + k) for k, n in enumerate(sizes)]
    solve(gpu_ctx, scene, clouds, [float(1.3 * n ** (-1.0 / 3.0)) for n in sizes], 12)


@pytest.mark.parametrize("n", [5640, 5641, 9200, 9201])
def test_largest_graphs(gpu_ctx, scene, n):
    solve(gpu_ctx, scene, [cloud(scene, n, 9)], [float(1.1 * n ** (-1.0 / 3.0))], 12, oracle=False)


def test_matrix_of_other_settings(gpu_ctx, scene):
    """Matrices marched under another cutoff or already solved keep to
    Floyd-Warshall: the same bits as with a schedule pinned."""
    import copy
    other = copy.deepcopy(scene.opts)
    other.cutoff = 0.02
    out = {}
    for schedule in (-1, 4):
        scenes.load_into(gpu_ctx, scene)
        gpu_ctx.set_fw_schedule(schedule)
        gpu_ctx.build_graphs([cloud(scene, 300, 5)], [np.float32(0.2) ** 2], 12)
        gpu_ctx.march_edges()
        gpu_ctx.set_settings(other)
        first = gpu_ctx.solve_paths(want=True)[0]
        used, _ = gpu_ctx.fw_schedule()
        out[schedule] = first, gpu_ctx.solve_paths(want=True)[0]
        assert used >= 0
    gpu_ctx.set_fw_schedule(-1)
    for a, b in zip(out[-1], out[4]):
        assert np.array_equal(a, b)
