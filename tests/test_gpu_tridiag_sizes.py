"""The batched tridiagonal solver at the edges of its forms: one layer, layers that do not fill a batch
of loads, the deepest system held in shared memory and the first that is not, one system, one more
than a block's, and a solve in place.  Diagonally dominant systems, condition below 10: the reference
sweep and this one each carry a few roundings a layer, well inside 1e-13."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def call(lib, n, m, t, out):
    from si3d_b200 import native
    native.check(lib.si3d_gpu_column_tridiag_noalloc(n, m, *[C.c_void_p(x.data_ptr()) for x in (*t, *out)], None))


@pytest.mark.parametrize("n,m", [(1, 5), (2, 33), (3, 1), (4, 64), (5, 31), (59, 40), (60, 33), (61, 33), (120, 65)])
def test_against_the_reference_sweep(native_libs, oracle_lib, n, m):
    import torch
    lib = native_libs.gpu()
    rng = np.random.default_rng(100 * n + m)
    a, c = -rng.uniform(0, 1, (n, m)), -rng.uniform(0, 1, (n, m))
    b = 2.2 + rng.uniform(0, 1, (n, m))
    a[0] = 0.0
    c[-1] = 0.0
    g, r = rng.standard_normal((n, m)), rng.standard_normal((n, m))
    t = [torch.from_numpy(x).cuda() for x in (a, b, c, g, r)]
    out = [torch.full((n, m), 7.0, dtype=torch.float64, device="cuda") for _ in range(2)]
    call(lib, n, m, t, out)
    got = [x.cpu().numpy() for x in out]
    for s in range(m):
        if n > 1:
            want = oracle_lib.trid(a[:, s], b[:, s], c[:, s], g[:, s], r[:, s])
        else:
            want = (g[:, s] / b[:, s], r[:, s] / b[:, s])
        for x, y in zip(got, want):
            np.testing.assert_allclose(x[:, s], y, rtol=1e-13, atol=1e-15)
    call(lib, n, m, t, t[3:])   # in place of the right-hand sides
    for x, y in zip(t[3:], out):
        assert torch.equal(x, y)
