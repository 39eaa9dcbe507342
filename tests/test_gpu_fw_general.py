"""The general path solve of one matrix (k_fw_panels, k_fw_update): directed
matrices at sizes around a panel block, an update tile, the padding and the line
between narrow and wide tiles, from host memory (padded) and in device memory
(ragged, with a leading dimension of its own). Against the FP32 oracle, 1e-6
relative as the FP32 min-plus elsewhere; both forms give the same bits."""
import ctypes as C

import numpy as np
import pytest

from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


def matrix(n, seed):
    rng = np.random.default_rng(seed)
    m = (rng.random((n, n), np.float32) * 3.0 + 0.01).astype(np.float32)
    m[rng.random((n, n)) > max(0.03, 6.0 / n)] = np.inf
    return m


@pytest.mark.parametrize("n", [1, 3, 63, 64, 65, 127, 128, 129, 191, 193, 257, 640, 1024, 1025])
def test_sizes(gpu_ctx, n):
    import torch
    m = matrix(n, n)
    got = gpu_ctx.fw_host(m)
    ref = po.fw_minplus_f32(m)
    assert np.array_equal(np.isfinite(got), np.isfinite(ref))
    f = np.isfinite(ref)
    assert np.allclose(got[f], ref[f], rtol=1e-6, atol=0.0)
    # in device memory: whole rows behind the matrix and columns beside it stay
    ld = (n + 3) // 4 * 4 + 4
    dev = torch.full((n + 2, ld), -1.0, device="cuda")
    dev[:n, :n] = torch.from_numpy(m)
    torch.cuda.synchronize()
    assert gpu_ctx.lib.lg_fw_device(C.c_void_p(dev.data_ptr()), n, ld, None) == 0
    out = dev.cpu().numpy()
    assert np.array_equal(out[:n, :n], got)
    assert (out[n:] == -1.0).all() and (out[:, n:] == -1.0).all()
