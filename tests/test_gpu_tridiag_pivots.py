"""The batched tridiagonal solver divides by each pivot: bit for bit the recurrence with three quotients a
layer, also for pivots so small that their reciprocal is not a number of the type."""
import numpy as np
import pytest

from test_gpu_tridiag_sizes import call

pytestmark = pytest.mark.gpu


def recurrence(a, b, c, g, r):
    n = len(b)
    ag, ar, e = np.empty_like(g), np.empty_like(r), np.empty_like(c)
    cp = dp = ep = np.zeros(b.shape[1])
    for k in range(n):
        den = b[k] if k == 0 else b[k] - a[k] * cp
        gk, rk = (g[k], r[k]) if k == 0 else (g[k] - a[k] * dp, r[k] - a[k] * ep)
        cp, dp, ep = c[k] / den, gk / den, rk / den
        e[k], ag[k], ar[k] = cp, dp, ep
    for k in range(n - 2, -1, -1):
        ag[k] = ag[k] - e[k] * ag[k + 1]
        ar[k] = ar[k] - e[k] * ar[k + 1]
    return ag, ar


@pytest.mark.parametrize("exponent", [0, -1027])   # -1027: pivots of 2 to 3e-309
@pytest.mark.parametrize("n,m", [(1, 3), (7, 33), (60, 40), (61, 40)])
def test_quotients_are_exact(native_libs, n, m, exponent):
    import torch
    lib = native_libs.gpu()
    rng = np.random.default_rng(10 * n + m)
    a, c = -rng.uniform(0, 1, (n, m)), -rng.uniform(0, 1, (n, m))
    b = 3.2 + rng.uniform(0, 1, (n, m))
    a[0] = 0.0
    c[-1] = 0.0
    g, r = rng.standard_normal((n, m)), rng.standard_normal((n, m))
    t = [np.ldexp(x, exponent) for x in (a, b, c, g, r)]
    if exponent:
        assert (1.0 / t[1] == np.inf).any()
    out = [torch.zeros((n, m), dtype=torch.float64, device="cuda") for _ in range(2)]
    call(lib, n, m, [torch.from_numpy(x).cuda() for x in t], out)
    for x, y in zip(out, recurrence(*t)):
        np.testing.assert_array_equal(x.cpu().numpy(), y)
