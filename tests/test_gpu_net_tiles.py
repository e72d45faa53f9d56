"""Gradient of the network at the edges of the 32 -> 32 weight gradient's tiles, 4 x 16 pixels: one row or column
fewer than a tile, a whole one, one more; tolerance as for the other gradient tests."""
import numpy as np
import pytest

from test_gpu_learn import _case, _gpu_net, _groups

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h", [3, 4, 5])
@pytest.mark.parametrize("w", [15, 16, 17])
def test_gradients_at_weight_gradient_tiles(native_libs, oracle_lib, h, w):
    p, feat, target, mask = _case(40 + h, 2, h, w)
    mask[:, 0, 0] = 1.0
    feat[..., 3] = mask
    out, loss, g = _gpu_net(native_libs, p, feat, target, mask)
    loss_ref, g_ref = oracle_lib.net_grad(p, feat, target, mask, bf16=True)
    assert loss == pytest.approx(loss_ref, rel=2e-2)
    for name, (a, b) in _groups().items():
        assert np.linalg.norm(g[a:b] - g_ref[a:b]) <= 3e-2 * np.linalg.norm(g_ref[a:b]), name
