"""A basin's columns numbered otherwise than row by row: the same fd call gives the same fields."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_parity import STATE_2D, STATE_3D, STATE_I

pytestmark = pytest.mark.gpu

MAPS = ("lEC", "lWC", "lNC", "lSC")


class Basin:
    """State, maps and depths of a run, and handles on them with the columns in another order."""

    def __init__(self, native, path):
        from si3d_b200.model import GpuRun
        self.native, self.lib = native, native.gpu()
        run = GpuRun(path, pcg_itmax=2000)
        try:
            self.im1, self.jm1, self.km1, self.lm = run.im1, run.jm1, run.km1, run.lm
            self.depth = {n: run.get(f).sum(axis=0) for n, f in (("hhs", "h"), ("hhu", "hu"), ("hhv", "hv"))}
            self.maps = {n: run.map(n) for n in (*MAPS, "l2i", "l2j", "kmz")}
            self.zlevel = np.empty(run.km1)
            native.check(run.h.si3d_host_get_zlevel(run.hm, native.ptr(self.zlevel)))
            run.run(3)
            self.state = {f: run.get(f) for f in STATE_3D + STATE_2D + list(STATE_I)}
        finally:
            run.close()

    def handle(self, new):
        """new[l]: the 0-based new number of 0-based column l; the last column, dry, stays."""
        old = np.argsort(new)
        m = {n: np.ascontiguousarray(a[old]) for n, a in self.maps.items()}
        for n in MAPS:
            m[n] = (new[m[n] - 1] + 1).astype(np.int32)
        d = {n: np.ascontiguousarray(a[old]) for n, a in self.depth.items()}
        ip, dp = (lambda a: a.ctypes.data_as(C.POINTER(C.c_int))), (lambda a: a.ctypes.data_as(C.POINTER(C.c_double)))
        nat = self.native
        g = nat.Grid(self.im1, self.jm1, self.km1, 2, self.lm, ip(m["l2i"]), ip(m["l2j"]), *[ip(m[n]) for n in ("lEC", "lWC", "lNC", "lSC")],
                     ip(m["kmz"]), dp(d["hhs"]), dp(d["hhu"]), dp(d["hhv"]), dp(self.zlevel))
        p = nat.Params(dt=30, dx=50, dy=50, Av0=1e-3, Dv0=1e-3, Ax0=1, Ay0=1, f=1e-4, theta=0.6, cd=0.0025, cw=1.2e-3,
                       beta=0.1, iadv=1, itrmom=1, ihd=1, ibc=1, isal=1, itrap=1, niter=2, pcg_test=5, pcg_tol=1e-12,
                       pcg_itmax=2000, srelpr=2.220446049250313e-16, ordering=1)
        h = C.c_int(-1)
        nat.check(self.lib.si3d_gpu_init(C.byref(g), C.byref(p), 0, C.byref(h)))
        for f, a in self.state.items():
            v = np.asfortranarray(a[..., old])
            nat.check((self.lib.si3d_gpu_set_ifield if f in STATE_I else self.lib.si3d_gpu_set_field)(h, f.encode(), nat.ptr(v)))
        return h

    def fields(self, h, new):
        out = {}
        for f, a in self.state.items():
            v = np.empty_like(a, order="F")
            self.native.check((self.lib.si3d_gpu_get_ifield if f in STATE_I else self.lib.si3d_gpu_get_field)(h, f.encode(), self.native.ptr(v)))
            out[f] = v[..., new]
        return out

    def launches(self, h):
        n = C.c_longlong(0)
        self.native.check(self.lib.si3d_gpu_counters(h, C.byref(n), None, None))
        return n.value


@pytest.fixture(scope="module")
def basin(native_libs, tmp_path_factory):
    from si3d_b200 import synth
    d = str(tmp_path_factory.mktemp("numbering"))
    nx, ny = 260, 210   # 300 tiles of faces and more in the natural order
    depth = synth.random_bathymetry(nx, ny, 77, corr=12.0, dmax=14.0)
    u = synth.wind_speed_for_stress(synth.stress_field(nx, ny, 78, corr=12.0))
    synth.write_run(synth.Basin("lake", nx, ny, 50.0, 50.0, depth, 14, 1.0, 30.0, 100, dzmin=0.1, uair=u, vair=0.2 * u), d)
    return Basin(native_libs, d)


def test_fd_in_another_numbering(native_libs, basin):
    """By columns of the grid and shuffled, against row by row: the zeta solve's sums run in another order,
    so the fields agree to its tolerance.  Shuffled, a face shares no neighbours with the next: its tiles hold
    a fraction of their faces, and the momentum stage keeps to the split kernels (7 launches in place of 5)."""
    n, rng = basin.lm, np.random.default_rng(3)
    i, j = basin.maps["l2i"][:n], basin.maps["l2j"][:n]
    by_columns, shuffled = np.empty(n, int), rng.permutation(n)
    by_columns[np.lexsort((i, j))] = np.arange(n)
    got, launched = [], []
    for order in (np.arange(n), by_columns, shuffled):
        new = np.append(order, n)
        h = basin.handle(new)
        try:
            before = basin.launches(h)
            basin.native.check(basin.lib.si3d_gpu_fd(h, 4, 1, 0, C.byref(basin.native.StepStats())))
            launched.append(basin.launches(h) - before)
            got.append(basin.fields(h, new))
        finally:
            basin.lib.si3d_gpu_finalize(h)
    assert launched == [24, 24, 26]
    for other in got[1:]:
        for f, a in got[0].items():
            if f in STATE_I:
                np.testing.assert_array_equal(other[f], a, err_msg=f)
            else:
                assert np.abs(other[f] - a)[..., :n].max() <= 1e-9 * max(np.abs(a).max(), 1e-300), f
