"""A graph with the diagonal neighbours of a grid everywhere but at a seam: the loop on the black unknowns, which
would merge the two ways to a diagonal neighbour, has to leave it to the two-colour loop."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def moebius(nx, ny, seed):
    """A strip of nx x ny nodes whose last row's east is its first row's, turned over: at the seam the node
    west of south is not the one south of west.  nx - ny is odd, so that the graph has two colours."""
    idx = np.arange(1, nx * ny + 1).reshape(nx, ny)
    east = np.concatenate([idx[1:], idx[:1, ::-1]]).ravel()
    west = np.concatenate([idx[-1:, ::-1], idx[:-1]]).ravel()
    dry = np.zeros((nx, 1), int)
    north = np.concatenate([idx[:, 1:], dry], axis=1).ravel()
    south = np.concatenate([dry, idx[:, :-1]], axis=1).ravel()
    jco = np.stack([idx.ravel(), west, south, north, east], 1).astype(np.int32)
    rng = np.random.default_rng(seed)
    sx, sy = rng.uniform(3, 30, nx * ny), rng.uniform(3, 30, nx * ny) * (north > 0)
    at = lambda s, n: np.where(n > 0, s[n - 1], 0.0)  # noqa: E731
    coef = np.stack([1 + sx + at(sx, west) + sy + at(sy, south), -at(sx, west), -at(sy, south), -sy, -sx], 1)
    x = rng.standard_normal(nx * ny)
    b = coef[:, 0] * x
    for m in range(1, 5):
        b += coef[:, m] * np.where(jco[:, m] > 0, x[jco[:, m] - 1], 0.0)
    return coef, jco, b, x


@pytest.mark.parametrize("precision", ["FP64", "MIXED_IR"])
@pytest.mark.parametrize("nx,ny", [(12, 9), (40, 33)])
def test_a_seam_that_does_not_close(native_libs, nx, ny, precision):
    from si3d_b200.model import solve_zeta
    coef, jco, b, x = moebius(nx, ny, nx)
    n = nx * ny
    assert n // 2 >= 32   # enough nodes of a colour for the loop on the black unknowns
    west, south = jco[:, 1], jco[:, 2]
    both = np.nonzero((west > 0) & (south > 0))[0]
    ws, sw = west[south[both] - 1], south[west[both] - 1]
    parity = np.add.outer(np.arange(nx), np.arange(ny)).ravel()[both] % 2
    differ = (ws > 0) & (sw > 0) & (ws != sw)
    assert differ[parity == 0].any() and differ[parity == 1].any()
    # with the two merged, the Schur complement of either colour would not be this matrix's
    A = np.zeros((n, n))
    for m in range(5):
        on = jco[:, m] > 0
        A[np.nonzero(on)[0], jco[on, m] - 1] += coef[on, m]
    assert np.array_equal(A, A.T) and np.abs(A @ x - b).max() < 1e-10
    got, info = solve_zeta(coef, jco, b, np.zeros(n), itmax=2000, precision=getattr(native_libs, f"SI3D_{precision}"))
    assert info["ier"] == 0 and info["stptst"] < 1e-12
    assert np.linalg.norm(got - x) <= 1e-12 * np.linalg.norm(b) + 8 * 2.2e-16 * 240.0 * np.linalg.norm(x)
