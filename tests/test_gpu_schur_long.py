"""The zeta solve's loop on the black unknowns in basins that are long along the numbering's fast index:
its window form gives way to the streaming one where the neighbours' nodes are many."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_schur import system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["FP64", "MIXED_IR"])
@pytest.mark.parametrize("nx,ny", [(10, 1000), (13, 1500), (14, 2000), (40, 3001), (2, 4000)])
def test_manufactured_solutions(native_libs, nx, ny, precision):
    """Both sides of the rule (reach 1000 to 3001, 495 to 510 nodes a block) and a cluster; tolerance as
    for the other shapes."""
    from si3d_b200.model import solve_zeta
    coef, jco, b, x = system(nx, ny, 0.02, seed=ny)
    got, info = solve_zeta(coef, jco, b, np.zeros_like(b), itmax=4000, precision=getattr(native_libs, f"SI3D_{precision}"))
    assert info["ier"] == 0 and info["stptst"] < 1e-12
    assert np.linalg.norm(got - x) <= 1e-12 * np.linalg.norm(b) + 8 * 2.2e-16 * 240.0 * np.linalg.norm(x)


def iteration_us(native, nx, ny, precision):
    """Device time of a CG iteration on a full nx x ny rectangle of one layer."""
    lib = native.gpu()
    lm = nx * ny
    idx = np.full((nx + 2, ny + 2), lm + 1, dtype=np.int32)
    idx[1:-1, 1:-1] = np.arange(1, lm + 1).reshape(nx, ny)
    i, j = (a.astype(np.int32) for a in np.nonzero(idx <= lm))
    E, W, N, S = (np.ascontiguousarray(idx[a, b]) for a, b in ((i + 1, j), (i - 1, j), (i, j + 1), (i, j - 1)))
    rng = np.random.default_rng(9)
    f = {n: np.zeros(lm + 1) for n in ("sx", "sy", "rr", "qq", "sp")}
    f["sx"][:lm] = rng.uniform(3, 30, lm) * (E <= lm)
    f["sy"][:lm] = rng.uniform(3, 30, lm) * (N <= lm)
    f["rr"][:lm] = 1 + f["sx"][:lm] + f["sx"][W - 1] * (W <= lm) + f["sy"][:lm] + f["sy"][S - 1] * (S <= lm)
    f["qq"][:lm] = rng.standard_normal(lm)
    kmz = np.full(lm + 1, 2, np.int32)
    kmz[lm] = 3
    one, zl = np.ones(lm + 1), np.array([-100.0, -100.0, 1.0])
    ip, dp = (lambda a: a.ctypes.data_as(C.POINTER(C.c_int))), (lambda a: a.ctypes.data_as(C.POINTER(C.c_double)))
    g = native.Grid(nx + 2, ny + 2, 3, 2, lm, ip(i), ip(j), ip(E), ip(W), ip(N), ip(S), ip(kmz), dp(one), dp(one), dp(one), dp(zl))
    p = native.Params(dt=1, dx=1, dy=1, theta=1, itrmom=1, ihd=1, pcg_test=5, pcg_tol=1e-12, pcg_itmax=500,
                      srelpr=2.2e-16, ordering=1, precision=precision)
    h = C.c_int(-1)
    native.check(lib.si3d_gpu_init(C.byref(g), C.byref(p), 0, C.byref(h)))
    try:
        top = np.full(lm + 1, 2, np.int32)
        for n in ("k1z", "k1u", "k1v"):
            native.check(lib.si3d_gpu_set_ifield(h, n.encode(), native.ptr(top)))
        for n, a in f.items():
            native.check(lib.si3d_gpu_set_field(h, n.encode(), native.ptr(a)))
        best = np.inf
        for _ in range(5):
            st, ms, cnt = native.StepStats(), np.zeros(16), np.zeros(16, np.int64)
            native.check(lib.si3d_gpu_profile(h, 1))
            native.check(lib.si3d_gpu_stage(h, b"solve", 1, C.byref(st)))
            assert st.ier[0] == 0
            native.check(lib.si3d_gpu_counters(h, None, native.ptr(ms), native.ptr(cnt)))
            k = native.STAGES.index("pcg_iter")
            best = min(best, 1e3 * ms[k] / cnt[k])
        return best
    finally:
        lib.si3d_gpu_finalize(h)


def test_a_turned_basin_takes_about_as_long(native_libs):
    """30 x 8000 and 8000 x 30 are the same work; polling a halo of 16000 nodes took three times as long."""
    native = native_libs
    long_way = iteration_us(native, 30, 8000, native.SI3D_MIXED_IR)
    assert long_way <= 2.0 * iteration_us(native, 8000, 30, native.SI3D_MIXED_IR)
