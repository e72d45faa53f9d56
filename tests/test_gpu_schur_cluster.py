"""The loop on the black unknowns as one cluster, at the edges of its range: two blocks with one node in
the second, eight full blocks (4096 black nodes), nine blocks (the grid's barriers again), single rows
(a halo of many blocks' nodes) and random numberings (a halo of every node, and one too wide for it).

Tolerance as for the loop's other sizes: the system's smallest eigenvalue is at least 1, so a solution
at relative residual 1e-12 is within 1e-12 |b| of the true one, plus the rounding of the residual."""
import numpy as np
import pytest

from test_gpu_schur import system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["FP64", "MIXED_IR"])
@pytest.mark.parametrize("nx,ny,land,order", [
    (27, 38, 0.0, None), (128, 64, 0.0, None), (128, 65, 0.0, None), (3000, 1, 0.0, None), (2, 1500, 0.0, None),
    (60, 50, 0.4, None), (40, 40, 0.0, 7), (110, 70, 0.0, 8)])
def test_cluster_sizes(native_libs, nx, ny, land, order, precision):
    from si3d_b200.model import solve_zeta
    coef, jco, b, x = system(nx, ny, land, seed=nx * 1000 + ny, order=order)
    got, info = solve_zeta(coef, jco, b, np.zeros_like(b), itmax=4000, precision=getattr(native_libs, f"SI3D_{precision}"))
    assert info["ier"] == 0 and info["stptst"] < 1e-12
    tol = 1e-12 * np.linalg.norm(b) + 8 * 2.2e-16 * 240.0 * np.linalg.norm(x)
    assert np.linalg.norm(got - x) <= tol
