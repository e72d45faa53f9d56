"""The network's gradient where the output gradient is far below one or values are infinite: it has to
be what FP32 multiply-adds give."""
import numpy as np
import pytest

from test_gpu_learn import _case, _groups

pytestmark = pytest.mark.gpu

B, H, W = 3, 8, 32   # whole tiles of the weight-gradient kernels: no padding pixel meets an infinity


def gradient(net, feat, gout):
    from si3d_b200 import native
    p = net._ptr
    native.check(net.g.si3d_net_backward(p(net.p), p(feat), p(gout), B, H, W, p(net.grad), p(net.ws), net.ws.numel()))
    return net.grad.cpu().numpy().astype(np.float64)


@pytest.mark.parametrize("exponent", [-60, -100, -105])
def test_tiny_output_gradients(native_libs, exponent):
    """The gradient is linear in the output's gradient, and a power of two changes no mantissa.  What may
    be lost is below 2^-149 (a product or a sum in FP32) or 2^-147 (the split's last term) a product: with
    768 pixels and values of X below 2^6 less than 768 * 2^-141 < 2^-131 in an entry."""
    import torch
    from si3d_b200.learn import Net
    p, feat, target, mask = _case(31, B, H, W)
    net = Net(B, H, W, p)
    f = torch.from_numpy(feat).to(net.dev)
    net.forward(f)
    rng = np.random.default_rng(5)
    gout = (rng.choice([-1.0, 1.0], (B, H, W)) * rng.uniform(1.0, 2.0, (B, H, W))).astype(np.float32)
    gout = torch.from_numpy(gout).to(net.dev)
    want = gradient(net, f, gout)
    got = gradient(net, f, gout * 2.0 ** exponent) * 2.0 ** -exponent
    assert np.abs(got - want).max() <= 2.0 ** (-131 - exponent)


def positive_net(stem_bias):
    """A network of positive weights: every pre-activation of positive features is positive."""
    from si3d_b200 import native
    rng = np.random.default_rng(7)
    p = rng.uniform(0.005, 0.01, native.NET_NPARAM).astype(np.float32)
    p[9 * 4 * 32] = stem_bias
    return p, rng.uniform(0.5, 1.5, (B, H, W, 4)).astype(np.float32), rng.uniform(1.0, 2.0, (B, H, W)).astype(np.float32)


def test_infinite_activation(native_libs):
    """One channel of the stem beyond BF16's range: infinite in every pixel, and so are all channels of the
    layers after it.  A finite positive gradient against it gives +infinity and against the stem's other
    channels the finite sums."""
    import torch
    from si3d_b200.learn import Net
    p, feat, gout = positive_net(3.4e38)
    net = Net(B, H, W, p)
    f = torch.from_numpy(feat).to(net.dev)
    net.forward(f)
    g = gradient(net, f, torch.from_numpy(gout).to(net.dev))
    groups = _groups()
    for k in range(4):
        w = g[groups[f"block{k}"][0]:][:9 * 32 * 32].reshape(9, 32, 32)
        assert (w[:, 0] == np.inf).all()
        assert (w[:, 1:] == np.inf).all() if k > 0 else (np.isfinite(w[:, 1:]).all() and (w[:, 1:] > 0).all())


def test_infinite_output_gradient(native_libs):
    """An infinite gradient at pixel row 4 of 0 .. 7: the weights of the 32 -> 32 layers get +infinity.  It
    spreads by a row a layer, to rows 3 .. 5 in the last layer, 1 .. 7 and 0 .. 7 in the first two; from the
    image's first and last row the taps beyond meet the zeros outside: NaN."""
    import torch
    from si3d_b200.learn import Net
    p, feat, gout = positive_net(0.01)
    net = Net(B, H, W, p)
    f = torch.from_numpy(feat).to(net.dev)
    net.forward(f)
    gout[1, 4, 13] = np.inf
    g = gradient(net, f, torch.from_numpy(gout).to(net.dev))
    for k in range(4):
        w = g[_groups()[f"block{k}"][0]:][:9 * 32 * 32].reshape(3, 3 * 32 * 32)   # rows of taps
        for row in range(3):
            outside = (row == 0 and k == 0) or (row == 2 and k <= 1)
            assert np.isnan(w[row]).all() if outside else (w[row] == np.inf).all()
