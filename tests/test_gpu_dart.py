"""GPU dart throwing (lg_scatter_points / lg_scatter_graphs) against the
oracle's scatterPoints, which runs the C++ library's std::mt19937 as the
reference's RandGen does: the accepted point sets must be identical (same
points, bit for bit, in the same order) and so must the connect radii."""
import numpy as np
import pytest

from lightgraph_gb300 import _capi, lightgraph as lgm, scenes
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


def connect_r2(m2, mult):
    r = np.sqrt(np.float32(m2)) * np.float32(mult)
    return np.float32(r * r)


def check_iterations(ctx, sc, opts, first, n):
    pts, r2 = ctx.scatter_points(first, n, opts)
    opt, ocnt, om2 = po.scatter_points(sc.density, opts, first, n)
    for i in range(n):
        assert len(pts[i]) == ocnt[i], (first + i, len(pts[i]), ocnt[i])
        assert np.array_equal(pts[i].view(np.uint32), opt[i, :ocnt[i]].view(np.uint32)), first + i
        assert np.float32(r2[i]) == connect_r2(om2[i], opts.connect_mult), first + i
    return pts, r2


def test_scatter_points_match_oracle(gpu_ctx):
    sc = scenes.small(n_points=16)
    scenes.load_into(gpu_ctx, sc)
    opts = lgm.scatter_opts(scatter_count=200000)
    check_iterations(gpu_ctx, sc, opts, 0, 4)
    check_iterations(gpu_ctx, sc, opts, 37, 2)


def test_scatter_points_reference_constants(gpu_ctx):
    sc = scenes.small(n_points=16)
    scenes.load_into(gpu_ctx, sc)
    opts = lgm.scatter_opts()
    assert opts.scatter_count == 1000000 and opts.target_size == 750
    pts, _ = check_iterations(gpu_ctx, sc, opts, 0, 1)
    assert 100 < len(pts[0]) <= 751


def test_scatter_graphs_connects_like_oracle(gpu_ctx):
    sc = scenes.small(n_points=16)
    scenes.load_into(gpu_ctx, sc)
    opts = lgm.scatter_opts(scatter_count=150000)
    pts, r2 = gpu_ctx.scatter_points(0, 2, opts)
    cnt = gpu_ctx.scatter_graphs(0, 2, 12, opts)
    assert [len(p) for p in pts] == list(cnt)
    S_dev = gpu_ctx.march_edges(want=True)
    adj, _ = gpu_ctx.build_graphs(pts, r2, 12, want_adjacency=True)
    S_host = gpu_ctx.march_edges(want=True)
    o = po.Oracle(sc.density, sc.shader, sc.opts, sc.lights)
    for i in range(2):
        assert np.array_equal(S_dev[i], S_host[i])
        oadj, ne = o.build_graph(pts[i], float(r2[i]), 12)
        assert ne > 0
        assert np.array_equal(adj[i].astype(bool), oadj.astype(bool))


@pytest.mark.parametrize("kw, dtype, origin", [
    (dict(scatter_count=1663, n_estimates=3), 0, (0, 0, 0)),            # below one chunk of 1664 candidates
    (dict(scatter_count=1665, n_estimates=1665), 0, (0, 0, 0)),         # one past it; a radius update per candidate
    (dict(scatter_count=2 * 1664, n_estimates=7), 1, (0, 0, 0)),        # whole chunks; updates inside them
    (dict(scatter_count=30000, n_estimates=18, target_size=5, hard_limit=7), 0, (0, 0, 0)),  # ends early
    (dict(scatter_count=60000, target_size=4000, hard_limit=4096, min_dist_mult=0.01), 2, (0, 0, 0)),  # most points
    (dict(scatter_count=20000, min_dist_mult=3.0), 0, (0, 0, 0)),       # a radius over the whole box
    (dict(scatter_count=40000), 0, (3.7, -120.3, 1000.1)),              # bbmin far from a float; coarse index space
])
def test_scatter_points_chunk_edges(gpu_ctx, kw, dtype, origin):
    """Candidate counts around a chunk, radius updates inside and at its ends,
    the smallest and largest point limits, storage types and a far world
    origin: the oracle's points, bit for bit."""
    sc = scenes.small(n_points=16, res=64)
    v = sc.density.values
    if dtype == 1:
        v = v.astype(np.float16).astype(np.float32)
    elif dtype == 2:
        v = (v.view(np.uint32) & np.uint32(0xFFFF0000)).view(np.float32)  # exactly representable in BF16
    sc.density.values = np.ascontiguousarray(v)
    sc.density.world_origin = origin
    scenes.load_into(gpu_ctx, sc, dtype)
    opts = lgm.scatter_opts(**kw)
    pts, r2 = gpu_ctx.scatter_points(11, 3, opts)
    opt, ocnt, om2 = po.scatter_points(sc.density, opts, 11, 3)
    for i in range(3):
        assert len(pts[i]) == ocnt[i]
        assert np.array_equal(pts[i].view(np.uint32), opt[i, :ocnt[i]].view(np.uint32))
        # (an expected size of 0 makes the radius NaN, on both sides)
        assert np.array_equal(np.float32(r2[i]), connect_r2(om2[i], opts.connect_mult), equal_nan=True)


@pytest.mark.parametrize("kw", [
    dict(scatter_count=3327, n_estimates=4),                 # below one chunk of 3328 candidates
    dict(scatter_count=3 * 3328 + 1, n_estimates=1),         # as many chunks as slots, and one candidate
    dict(scatter_count=7 * 3328, n_estimates=7),             # a radius update at the end of every chunk
    dict(scatter_count=30000, n_estimates=18, target_size=5, hard_limit=7),  # ends early, helpers ahead
    dict(scatter_count=30000, target_size=4000, hard_limit=4096, min_dist_mult=0.01),
])
def test_scatter_points_batch_sizes(gpu_ctx, kw):
    """A cluster of three CTAs an iteration, of two, one CTA alone, and two to
    an SM, by the number of iterations: the same points bit for bit, the first
    and last the oracle's."""
    sc = scenes.small(n_points=16, res=64)
    scenes.load_into(gpu_ctx, sc)
    opts = lgm.scatter_opts(**kw)
    pts, r2 = gpu_ctx.scatter_points(3, 170, opts)
    for n in (1, 24, 45, 60, 76, 100):
        p, q = gpu_ctx.scatter_points(3, n, opts)
        assert np.array_equal(np.asarray(q), np.asarray(r2)[:n], equal_nan=True)
        for i in range(n):
            assert np.array_equal(p[i].view(np.uint32), pts[i].view(np.uint32)), (n, i)
    check_iterations(gpu_ctx, sc, opts, 3, 1)
    check_iterations(gpu_ctx, sc, opts, 172, 1)


@pytest.mark.parametrize("target", [1, 3, 9, 40, 200])
def test_early_ends_on_clusters(gpu_ctx, target):
    """Iterations that end while their helper CTAs are at every stage of the
    chunks ahead (18 of them): each helper leaves as a whole, and the points are
    those of one CTA alone."""
    sc = scenes.small(n_points=16, res=64)
    scenes.load_into(gpu_ctx, sc)
    opts = lgm.scatter_opts(scatter_count=60000, target_size=target, hard_limit=target + 2, min_dist_mult=0.2)
    alone, r2 = gpu_ctx.scatter_points(0, 100, opts)
    assert max(len(p) for p in alone) == target + 1
    for _ in range(8):
        for n in (50, 70):  # clusters of three and of two
            pts, q = gpu_ctx.scatter_points(0, n, opts)
            assert np.array_equal(np.asarray(q), np.asarray(r2)[:n], equal_nan=True)
            for i in range(n):
                assert np.array_equal(pts[i].view(np.uint32), alone[i].view(np.uint32)), (n, i)


def test_waits_between_ctas_give_up(gpu_ctx):
    """A cluster whose first CTA does not wait for the first chunk's words (one
    look at them) ends with an error and leaves the context usable; with the
    limit in use no wait runs out."""
    import ctypes
    sc = scenes.small(n_points=16, res=64)
    scenes.load_into(gpu_ctx, sc)
    opts = lgm.scatter_opts(scatter_count=60000)
    check = lambda polls: gpu_ctx.lib.lg_dart_wait_check(gpu_ctx.h, ctypes.byref(opts), polls)  # noqa: E731
    for _ in range(3):
        assert check(1) == _capi.LG_ERR_TIMEOUT
        assert b"ran out" in gpu_ctx.lib.lg_last_error(gpu_ctx.h)
        check_iterations(gpu_ctx, sc, opts, 0, 2)
    assert check(1 << 22) == _capi.LG_OK
    assert check(0) == _capi.LG_ERR_INVALID
    assert check((1 << 24) + 1) == _capi.LG_ERR_INVALID


def test_largest_candidate_counts(gpu_ctx):
    """Up to 2^32 - 1 candidates an iteration, which ends at its target."""
    sc = scenes.small(n_points=16, res=64)
    scenes.load_into(gpu_ctx, sc)
    for count in (2 ** 32 - 3328, 2 ** 32 - 3327, 2 ** 32 - 1):
        opts = lgm.scatter_opts(scatter_count=count, target_size=40, hard_limit=50, min_dist_mult=0.1)
        check_iterations(gpu_ctx, sc, opts, 0, 2)
