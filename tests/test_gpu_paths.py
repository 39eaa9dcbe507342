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


def rewired(sc, factor=1.0, span=0.0, step=None, **shader):
    """The scene with its extinction times factor, without dropout, its density
    falling by e^-span across the volume, marched in steps of `step` voxels."""
    import copy
    out = copy.copy(sc)
    out.shader, out.opts = copy.deepcopy(sc.shader), copy.deepcopy(sc.opts)
    out.shader.setScattering(tuple(factor * s for s in sc.shader.scattering))
    out.shader.setAbsorption(tuple(factor * a for a in sc.shader.absorption))
    for k, v in shader.items():
        setattr(out.shader, k, v)
    out.opts.cutoff = 0.0
    if step:
        out.opts.step = (1.0, step)
    if span:
        out.density = copy.copy(sc.density)
        fall = np.exp(-span * np.linspace(0.0, 1.0, sc.density.values.shape[2]))
        out.density.values = np.ascontiguousarray(sc.density.values * fall, np.float32)
    return out


def paths(ctx, sc, clouds, radius, schedule):
    scenes.load_into(ctx, sc)
    ctx.set_fw_schedule(schedule)
    ctx.build_graphs(clouds, [np.float32(radius) ** 2] * len(clouds), 12)
    S = ctx.march_edges(want=True)
    out = S, ctx.solve_paths(want=True), ctx.fw_schedule()[0]
    ctx.set_fw_schedule(-1)
    return out


@pytest.mark.parametrize("kw", [
    dict(), dict(factor=1e-2), dict(factor=1e-4), dict(factor=1e-6),     # thin volumes
    dict(factor=1000.0),                                                # no transmittance along most paths
    dict(scattering=(0.002, 0.1, 1.0)),                                 # channels far apart
    dict(step=4.0),                                                     # edges without a sample: depth 0
    dict(span=9.0, scatter_density_min=3e-5, density_max=1.0),          # densities and so depths far apart
    dict(scatter_density_min=3e-5, density_max=1.0, density_scale=0.01),  # many edges at the least density
])
@pytest.mark.parametrize("n, radius", [(503, 0.2), (2051, 0.11)])
def test_distances(gpu_ctx, scene, kw, n, radius):
    """The distances against FP64: as the FP32 oracle's within 1e-6 and finite
    where those are, off by no more than Floyd-Warshall's in the mean, and at
    most by five halves of an FP32 unit (one rounding of 2^-24, and as many as
    the longest sums differ by where two paths nearly tie)."""
    sc = rewired(scene, **kw)
    clouds = [cloud(scene, n, 11)]
    S, dist, used = paths(gpu_ctx, sc, clouds, radius, -1)
    assert used == -1  # from the edges
    S4, fw, _ = paths(gpu_ctx, sc, clouds, radius, 4)
    assert np.array_equal(S[0], S4[0])
    true = po.apsp_dijkstra_f64(S[0])
    np.fill_diagonal(true, 0.0)
    fin = np.isfinite(true)
    if n < 1000:
        ref = po.fw_minplus_f32(S[0])
        np.fill_diagonal(ref, 0.0)
        assert np.array_equal(np.isfinite(ref), fin)
        assert np.allclose(dist[0][fin], ref[fin], rtol=1e-6, atol=0)
    assert np.array_equal(np.isfinite(dist[0]), fin) and np.array_equal(dist[0], dist[0].T)
    on = fin & (true > 1e-30)
    if "step" in kw:
        assert np.sum(S[0] == 0.0) > n / 2 and np.any(on)  # both kinds of edges
    assert np.all(dist[0][fin & ~on] == 0.0)
    off = np.abs(dist[0][on] / true[on] - 1.0)
    off_fw = np.abs(fw[0][on] / true[on] - 1.0)
    print("PATHS", n, kw, "rms %.2e / %.2e max %.2e / %.2e" % (np.sqrt(np.mean(off ** 2)), np.sqrt(np.mean(off_fw ** 2)), off.max(), off_fw.max()))
    assert np.mean(off ** 2) <= np.mean(off_fw ** 2)
    assert off.max() <= 2.5 * 2.0 ** -23
    if kw.get("factor") == 1000.0:
        assert true[on].max() * min(-e for e in sc.shader.getExtinction()) > 400.0


def test_depths_too_far_apart(gpu_ctx, scene):
    """Depths that may lie further apart than 2^20: Floyd-Warshall, the same
    bits as with a schedule pinned, also where they were marched so and the
    settings have changed since."""
    for least in (0.0, 1e-6):
        sc = rewired(scene, span=9.0, scatter_density_min=least, density_max=10.0)
        clouds = [cloud(scene, 307, 12)]
        _, dist, used = paths(gpu_ctx, sc, clouds, 0.2, -1)
        assert used >= 0
        _, fw, _ = paths(gpu_ctx, sc, clouds, 0.2, 4)
        assert np.array_equal(dist[0], fw[0])
        scenes.load_into(gpu_ctx, sc)
        gpu_ctx.build_graphs(clouds, [np.float32(0.2) ** 2], 12)
        gpu_ctx.march_edges()
        later = rewired(scene, span=9.0)
        gpu_ctx.set_shader(later.shader)
        assert np.array_equal(gpu_ctx.solve_paths(want=True)[0], fw[0])


def test_diffusion_under_another_extinction(gpu_ctx, scene):
    """Radiances diffused again under a smaller extinction than that of the
    solve: as with a schedule pinned."""
    thick = rewired(scene, factor=1000.0)
    out = []
    for schedule in (-1, 4):
        scenes.load_into(gpu_ctx, thick)
        gpu_ctx.set_fw_schedule(schedule)
        gpu_ctx.build_graphs([cloud(scene, 400, 12)], [np.float32(0.2) ** 2], 12)
        gpu_ctx.solve_graphs()
        gpu_ctx.set_shader(rewired(scene, factor=0.1).shader)
        out.append(gpu_ctx.diffuse(want=True))
    gpu_ctx.set_fw_schedule(-1)
    assert np.allclose(out[0], out[1], rtol=1e-4, atol=1e-7) and out[1].max() > 0


def test_graphs_dealt_over_calls(gpu_ctx, scene):
    """Nine graphs in one call and dealt over two: the same radiances bit for bit
    with a schedule set, and to FP32 roundings (one call goes by Floyd-Warshall,
    the others from the edges) without."""
    sizes = [300, 120, 257, 64, 400, 90, 333, 210, 150]
    clouds = [cloud(scene, n, 20 + n) for n in sizes]
    r2 = [np.float32(1.3 * n ** (-1.0 / 3.0)) ** 2 for n in sizes]
    scenes.load_into(gpu_ctx, scene)
    for schedule in (4, 2, -1):
        gpu_ctx.set_fw_schedule(schedule)
        out = []
        for parts in ([slice(0, 9)], [slice(0, 1), slice(1, 9)]):
            D = []
            for part in parts:
                gpu_ctx.build_graphs(clouds[part], r2[part], 12)
                D.append(gpu_ctx.solve_graphs(want=True))
            out.append(np.concatenate(D))
        if schedule >= 0:
            assert np.array_equal(out[0], out[1]), schedule
        else:
            assert np.allclose(out[0], out[1], rtol=4e-6, atol=0)
    gpu_ctx.set_fw_schedule(-1)


def test_channels_far_apart(gpu_ctx, scene):
    """Radiances under extinctions a hundred times apart, as the oracle's."""
    solve(gpu_ctx, rewired(scene, scattering=(0.002, 0.1, 1.0), absorption=(0.001, 0.02, 0.1)),
          [cloud(scene, 301, 14)], [0.2], 12)
