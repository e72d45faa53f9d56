"""Gradient of the network at the sizes where the weight-gradient kernels' tiles (8 x 16 pixels, 296
blocks that stride over them) are cut: one pixel, less than a tile, one row or column more than a tile,
more tiles than blocks.  Tolerance: that of the gradient test at one size (the BF16 rounding points are
the oracle's; the order of the FP32 sums is not, which moves single roundings by 2^-9)."""
import numpy as np
import pytest

from test_gpu_learn import _case, _gpu_net, _groups

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 7, 15), (1, 9, 17), (3, 8, 33), (5, 129, 65)])
def test_gradients_at_tile_edges(native_libs, oracle_lib, shape):
    p, feat, target, mask = _case(21, *shape)
    mask[:, 0, 0] = 1.0
    feat[..., 3] = mask
    out, loss, g = _gpu_net(native_libs, p, feat, target, mask)
    loss_ref, g_ref = oracle_lib.net_grad(p, feat, target, mask, bf16=True)
    assert loss == pytest.approx(loss_ref, rel=2e-2)
    for name, (a, b) in _groups().items():
        num, den = np.linalg.norm(g[a:b] - g_ref[a:b]), np.linalg.norm(g_ref[a:b])
        assert num <= 3e-2 * den, (name, num / den)
