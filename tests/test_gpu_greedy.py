"""The graph build's two forms, by sweeps (k_pair_sweep) and row by row
(k_greedy), against the oracle's buildGraph: point counts around a warp, a
block and the limit between the forms, caps from one to the largest, partner
counts around the words of a state and the length of a list (96), and batches
in which only some graphs take one form."""
import numpy as np
import pytest

from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


def cloud(n, seed, side=1.0):
    rng = np.random.default_rng(seed)
    return ((rng.random((n, 3)) - 0.5) * side).astype(np.float32)


@pytest.mark.parametrize("cap", [1, 12, 95, 96, 255])
def test_sizes_and_caps(gpu_ctx, cap):
    sizes = [1, 2, 31, 32, 33, 127, 1023, 1024, 1025]
    clouds = [cloud(n, n) for n in sizes]
    # about 40 partners inside the radius; the last two share one dense cluster each
    r = [np.float32((40.0 / max(n, 40) * 0.24) ** (1.0 / 3.0)) for n in sizes]
    clouds += [np.concatenate([cloud(300, 5), cloud(97, 6, 0.01)]), cloud(98, 7, 0.01)]
    # all partners of one another: 255, 256 and 257 each; and 258 in a wider cloud
    clouds += [cloud(256, 8, 0.01), cloud(257, 9, 0.01), cloud(258, 10, 0.01),
               np.concatenate([cloud(700, 11), cloud(258, 12, 0.01)])]
    r += [np.float32(0.2)] * 6
    r2 = [x * x for x in r]
    adj, ne = gpu_ctx.build_graphs(clouds, r2, cap, want_adjacency=True)
    for g, p in enumerate(clouds):
        ref, ne_ref = po.build_graph(p, r2[g], cap)
        assert np.array_equal(adj[g], ref), (g, len(p))
        assert ne[g] == ne_ref


@pytest.mark.parametrize("n", [600, 4800, 4864, 4865])
def test_sparse_graphs(gpu_ctx, n):
    """Few partners a point, which is what the sweeps are for; past 4864 points
    in all, rows."""
    p = cloud(n, 3)
    r = np.float32((14.0 / n * 0.24) ** (1.0 / 3.0))
    r2 = r * r
    for cap in (1, 5, 12):
        adj, ne = gpu_ctx.build_graphs([p], [r2], cap, want_adjacency=True)
        ref, ne_ref = po.build_graph(p, r2, cap)
        assert np.array_equal(adj[0], ref) and ne[0] == ne_ref


@pytest.mark.parametrize("near", [95, 96, 97, 130])
def test_partners_below_overflow(gpu_ctx, near):
    """The last point has `near` partners, all before it, each of which has
    fewer than 96 after it; beside a graph that stays with the sweeps."""
    rng = np.random.default_rng(near)
    d = rng.normal(size=(near, 3))
    ball = d / np.linalg.norm(d, axis=1)[:, None] * (0.0099 * rng.random((near, 1)) ** (1.0 / 3.0))
    far = cloud(1500, 4, 2.0) + np.float32(3.0)
    p = np.concatenate([far, ball, np.zeros((1, 3))]).astype(np.float32)
    r2 = np.float32(0.01) * np.float32(0.01)
    q = cloud(700, 5)
    q2 = np.float32(0.13) * np.float32(0.13)
    for cap in (3, 200):
        adj, ne = gpu_ctx.build_graphs([p, q], [r2, q2], cap, want_adjacency=True)
        for g, (c, c2) in enumerate([(p, r2), (q, q2)]):
            ref, ne_ref = po.build_graph(c, c2, cap)
            assert np.array_equal(adj[g], ref) and ne[g] == ne_ref


def lattice_ball(n, partners):
    """A jittered lattice in a ball, in order of the distance from its centre."""
    rng = np.random.default_rng(2)
    m = np.arange(-14, 15)
    g = np.stack(np.meshgrid(m, m, m, indexing="ij"), -1).reshape(-1, 3) + rng.uniform(-0.2, 0.2, (29 ** 3, 3))
    near = np.argsort(np.linalg.norm(g, axis=1))[:n]
    return (g[near] * 0.05).astype(np.float32), np.float32(0.05 * (partners * 0.75 / np.pi) ** (1.0 / 3.0))


@pytest.mark.parametrize("n, partners, lists, below", [
    (4700, 200.0, (2048, 4700), (0, 96)),   # past 2047 lists overflow, and no list of partners below does
    (4700, 188.0, (1024, 2047), (0, 96)),
    (4096, 900.0, (2048, 4096), (97, 4096)),  # dense throughout
])
def test_many_lists_overflow(gpu_ctx, n, partners, lists, below):
    """Graphs in which more rows have more than 96 partners past them than a
    32-bit sum of 2^20 each could count."""
    from scipy.spatial import cKDTree
    p, r = lattice_ball(n, partners)
    pairs = cKDTree(p.astype(np.float64)).query_pairs(float(r), output_type="ndarray")
    over = (np.bincount(pairs.min(axis=1), minlength=n) > 96).sum()
    assert lists[0] <= over <= lists[1]
    assert below[0] <= np.bincount(pairs.max(axis=1), minlength=n).max() <= below[1]
    r2 = r * r
    for cap in (12, 100, 255):
        adj, ne = gpu_ctx.build_graphs([p], [r2], cap, want_adjacency=True)
        ref, ne_ref = po.build_graph(p, r2, cap)
        assert np.array_equal(adj[0], ref) and ne[0] == ne_ref, cap
