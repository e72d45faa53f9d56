"""Forward pass and gradient of the network at the sizes where the weight-gradient kernels' tiles (8 x 16 pixels, 296
blocks that stride over them) are cut: one pixel, less than a tile, one row or column more than a tile,
more tiles than blocks; for the forward convolution also the edge of its 4 x 128 pixel tile.
Tolerance: that of the forward and gradient tests (the BF16 rounding points are
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


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 4, 128), (1, 6, 131), (3, 3, 257)])
def test_forward_at_tile_edges(native_libs, oracle_lib, shape):
    p, feat, target, mask = _case(22, *shape)
    mask[:, 0, 0] = 1.0
    out, _, _ = _gpu_net(native_libs, p, feat, target, mask)
    ref = oracle_lib.net_forward(p, feat, bf16=True)
    scale = np.abs(ref).max()
    assert np.abs(out - ref).max() <= 2e-2 * scale
