"""The zeta solve's loop on the black unknowns at the sizes where it changes form: just too few nodes
for it (31 black ones) and just enough, single rows, blocks that are just full, more nodes a block
than registers hold, numberings whose window does not fit in shared memory (the form that streams z
and p), and a graph that is no plain grid (the two-colour loop).

The system's smallest eigenvalue is at least 1 (unit mass plus a graph Laplacian), so a solution at
relative residual 1e-12 is within 1e-12 |b| of the true one; the recursive residual drifts from the
true one by rounding, a few times the unit roundoff times the largest row sum (240) of |x|."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def system(nx, ny, land=0.0, ratio=30.0, seed=0, order=None):
    """Purdue arrays of a five-point system on an nx x ny grid with a share of land cells, a solution
    and its right-hand side; `order`: None for the grid's numbering, a seed for a random one."""
    rng = np.random.default_rng(seed)
    wet = rng.random((nx, ny)) >= land
    wet[0, 0] = True
    lm = int(wet.sum())
    num = np.arange(1, lm + 1)
    if order is not None:
        np.random.default_rng(order).shuffle(num)
    idx = np.zeros((nx + 2, ny + 2), dtype=np.int64)
    idx[1:-1, 1:-1][wet] = num
    c = rng.uniform(0.1 * ratio, ratio, (2, nx + 2, ny + 2))
    cx = c[0, :-1] * (idx[:-1] > 0) * (idx[1:] > 0)
    cy = c[1][:, :-1] * (idx[:, :-1] > 0) * (idx[:, 1:] > 0)
    i, j = np.nonzero(idx)
    sort = np.argsort(idx[i, j])
    i, j = i[sort], j[sort]
    e, w, n, s = cx[i, j], cx[i - 1, j], cy[i, j], cy[i, j - 1]
    jco = np.stack([idx[i, j], idx[i - 1, j], idx[i, j - 1], idx[i, j + 1], idx[i + 1, j]], 1).astype(np.int32)
    coef = np.stack([1 + e + w + n + s, -w, -s, -n, -e], 1)
    x = np.zeros((nx + 2, ny + 2))
    x[i, j] = rng.standard_normal(lm)
    b = (coef[:, 0] * x[i, j] + coef[:, 1] * x[i - 1, j] + coef[:, 2] * x[i, j - 1] + coef[:, 3] * x[i, j + 1] +
         coef[:, 4] * x[i + 1, j])
    return coef, jco, b, x[i, j].copy()


@pytest.mark.parametrize("precision", ["FP64", "MIXED_IR"])
@pytest.mark.parametrize("nx,ny,land,order", [
    (9, 7, 0.0, None), (8, 8, 0.0, None), (1, 90, 0.0, None), (90, 1, 0.0, None), (13, 11, 0.5, None),
    (32, 32, 0.0, None), (33, 31, 0.0, None), (41, 25, 0.3, None), (64, 33, 0.1, None),
    (601, 307, 0.3, None), (760, 650, 0.0, None),   # 760 x 650: 1669 nodes a block, 1536 in registers
    (300, 260, 0.2, 5),                             # random numbering: the window does not fit
])
def test_manufactured_solutions(native_libs, nx, ny, land, order, precision):
    from si3d_b200.model import solve_zeta
    coef, jco, b, x = system(nx, ny, land, seed=nx * 1000 + ny, order=order)
    got, info = solve_zeta(coef, jco, b, np.zeros_like(b), itmax=4000, precision=getattr(native_libs, f"SI3D_{precision}"))
    assert info["ier"] == 0 and info["stptst"] < 1e-12
    tol = 1e-12 * np.linalg.norm(b) + 8 * 2.2e-16 * 240.0 * np.linalg.norm(x)
    assert np.linalg.norm(got - x) <= tol


def test_iterations_match_the_oracle(native_libs, oracle_lib):
    """The loop on the black unknowns takes the iterations of the red-black MIC-CG it restates."""
    from si3d_b200.model import solve_zeta
    for nx, ny, land, x0 in ((33, 31, 0.0, 0.0), (64, 33, 0.1, 0.5), (80, 60, 0.3, 1.0)):
        coef, jco, b, x = system(nx, ny, land, seed=3)
        start = x0 * x + 0.01 * np.random.default_rng(4).standard_normal(x.size)
        _, o = oracle_lib.pcg(coef, jco, b, start, ordering=1, itmax=2000)
        _, g = solve_zeta(coef, jco, b, start, itmax=2000)
        assert abs(o["iters"] - g["iters"]) <= 1


def test_a_graph_that_is_no_grid(native_libs):
    """West of south and south of west differ: the two-colour loop solves it."""
    from si3d_b200.model import solve_zeta
    # a cycle of eight nodes, walked by E and N links alternately: 1 -E- 2 -N- 3 -E- 4 ... 8 -N- 1
    n = 8
    jco = np.zeros((n, 5), dtype=np.int32)
    coef = np.zeros((n, 5))
    jco[:, 0] = np.arange(1, n + 1)
    for k in range(0, n, 2):
        a, c, d = k, k + 1, (k + 2) % n
        jco[a, 4], jco[c, 1] = c + 1, a + 1            # a's east is c, c's west is a
        jco[c, 3], jco[d, 2] = d + 1, c + 1            # c's north is d, d's south is c
        coef[a, 4] = coef[c, 1] = -(3.0 + k)
        coef[c, 3] = coef[d, 2] = -(2.0 + k)
    coef[:, 0] = 1.0 - coef[:, 1:].sum(1)
    x = np.linspace(-1.0, 1.0, n)
    b = coef[:, 0] * x
    for m in range(1, 5):
        b += coef[:, m] * np.where(jco[:, m] > 0, x[np.maximum(jco[:, m], 1) - 1], 0.0)
    got, info = solve_zeta(coef, jco, b, np.zeros(n), itmax=100)
    assert info["ier"] == 0
    assert np.linalg.norm(got - x) <= 1e-12 * np.linalg.norm(b) + 1e-14
