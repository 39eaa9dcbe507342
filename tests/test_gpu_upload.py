"""Grid upload (k_pack_volume): boxes off the brick size, a single voxel, thin
boxes, explicit leaf masks, every storage type, checked through what the
records, bitmaps and bounds are used for: edge depths (1e-4 against the FP64
oracle, reachability exact) and the scatter grid's topology and values, with
coarse voxels inside, equal to and across bricks."""
import numpy as np
import pytest

from lightgraph_gb300.lightgraph import Grid, Light, SceneSettings, Shader
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


def quantised(v, dtype):
    if dtype == 1:
        return v.astype(np.float16).astype(np.float32)
    if dtype == 2:
        return (v.view(np.uint32) & np.uint32(0xFFFF0000)).view(np.float32)
    return v


@pytest.mark.parametrize("factor", [3, 4, 8, 16])
@pytest.mark.parametrize("dims, dtype, masked", [
    ((1, 1, 1), 0, False), ((9, 17, 8), 1, False), ((8, 8, 8), 2, True), ((33, 5, 40), 0, True), ((16, 24, 7), 0, False),
])
def test_boxes(gpu_ctx, dims, dtype, masked, factor):
    rng = np.random.default_rng(dims[0] * 100 + dims[1])
    nx, ny, nz = dims
    v = (rng.random((nz, ny, nx)) * 0.8 + 0.1).astype(np.float32)
    v[rng.random((nz, ny, nx)) < 0.5] = 0.0
    v[0, 0, 0] = 0.5
    v[nz // 2:, :, :nx // 2] = 0.0  # empty bricks beside full ones
    v = np.ascontiguousarray(quantised(v, dtype))
    leaves = tuple((n + 7) // 8 for n in (nz, ny, nx))
    mask = (rng.random(leaves) < 0.7).astype(np.uint8) if masked else None
    if masked:
        mask[0, 0, 0] = 1
    g = Grid(v, (-8, 0, 16), 0.1, leaf_mask=mask)
    sh = Shader()
    opts = SceneSettings(width=8, height=8, step=(1.0, 0.25), iter=1, scatterGridResFactor=factor)
    lights = [Light.parse("dir:0:1,1,1:1.0:-35,25,0")]
    gpu_ctx.upload_density(g, dtype)
    gpu_ctx.upload_temperature(None)
    gpu_ctx.set_shader(sh)
    gpu_ctx.set_settings(opts)
    gpu_ctx.set_lights(lights)
    lo = np.array([-8, 0, 16]) * 0.1
    pts = (lo + rng.random((60, 3)) * (np.array(dims) * 0.1)).astype(np.float32)
    r2 = np.float32(max(dims) * 0.05) ** 2
    adj, _ = gpu_ctx.build_graphs([pts], [r2], 12, want_adjacency=True)
    S = gpu_ctx.march_edges(want=True)[0]
    o = po.Oracle(g, sh, opts, lights)
    _, ref = o.march_edges(pts, adj[0], want_T=False)
    fin = np.isfinite(ref)
    assert np.array_equal(np.isfinite(S), fin)
    assert np.allclose(S[fin], ref[fin], rtol=1e-4, atol=1e-6)
    D = gpu_ctx.solve_graphs(want=True)
    gpu_ctx.splat()
    clo, cdims, vals = gpu_ctx.scatter_grid()
    rlo, rdims, rvals, _ = o.splat(pts, D)
    assert clo == rlo and cdims == rdims
    assert np.array_equal(vals != 0, rvals != 0)
    assert np.allclose(vals, rvals, rtol=1e-4, atol=1e-7)


def test_staging_is_given_back():
    """After an upload a context holds the records, the bitmaps and at most 64 MB
    of staging, whatever the size of the grid."""
    import torch
    from lightgraph_gb300 import Context
    ctx = Context(0)
    ctx.upload_density(Grid(np.ones((8, 8, 8), np.float32), (0, 0, 0), 0.1), 1)  # first-use allocations
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    n = 416  # 288 MB of staging
    ctx.upload_density(Grid(np.ones((n, n, n), np.float32), (0, 0, 0), 0.1), 1)
    held = free - torch.cuda.mem_get_info()[0]
    records = (n // 8 + 2) ** 3 * 512 * 16
    ctx.close()
    assert held <= records + (96 << 20)
