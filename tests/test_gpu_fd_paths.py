"""Paths of fd that its stage calls do not take: the copies of the surface layer stage that fd leaves
out (the state must end as after the stage-by-stage calls, which make them), and continuity with one
thread per column, used from 65536 columns on."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = "h hp hpp wp uh uhp uhpp up upp hu hup hupp agx arx vh vhp vhpp vp vpp hv hvp hvpp agy ary Bth2 Bth3 Bth4".split()
OTHER = "sal salp salpp rhop Av Dv".split()


@pytest.mark.parametrize("name", ["t0", "t1"])
def test_fd_ends_as_its_stages_do(native_libs, run_dirs, name):
    from si3d_b200 import native
    from si3d_b200.model import GpuRun
    a = GpuRun(run_dirs[name], pcg_itmax=2000)
    b = GpuRun(run_dirs[name], pcg_itmax=2000)
    try:
        a.run(3)
        b.run(3)
        st = native.StepStats()
        native.check(a.g.si3d_gpu_fd(a.gh, 4, 1, 0, C.byref(st)))
        for s in ("momentum", "matcon", "solve", "vel", "scalar", "vel2"):
            b.stage(s, 1)
        for f in FIELDS + OTHER:
            np.testing.assert_array_equal(a.get(f), b.get(f), err_msg=f)
    finally:
        a.close()
        b.close()


@pytest.mark.parametrize("nx,ny", [(270, 260), (520, 140)])
def test_one_thread_per_column_continuity(native_libs, tmp_path, nx, ny):
    """More than 65536 wet columns: wp against the layer sums of the same state (the recurrence of
    continuity(2), in the same order)."""
    from si3d_b200 import synth
    from si3d_b200.model import GpuRun
    rng = np.random.default_rng(nx)
    depth = np.round(rng.uniform(1.0, 5.0, (nx, ny)), 1)
    d = str(tmp_path / "lake")
    u = 4.0 + rng.uniform(-1.0, 1.0, (nx, ny))
    synth.write_run(synth.Basin("lake", nx, ny, 100.0, 100.0, depth, 5, 1.0, 20.0, 100, dzmin=0.1, uair=u, vair=0.0 * u), d)
    g = GpuRun(d, pcg_itmax=4000)
    try:
        assert g.lm >= 65536
        g.run(3)
        uhp, vhp, wp, k1z, kmz = g.get("uhp"), g.get("vhp"), g.get("wp"), g.get("k1z"), g.map("kmz")
        lW, lS = g.map("lWC"), g.map("lSC")
        w = np.zeros(g.lm)
        want = np.zeros((g.km1, g.lm))
        m = np.arange(g.lm)
        for k in range(g.km1, 1, -1):
            i = k - 1
            on = (k <= kmz[m]) & (k >= k1z[m])
            w = np.where(on, w - (uhp[i, m] - uhp[i, lW[m] - 1]) / 100.0 - (vhp[i, m] - vhp[i, lS[m] - 1]) / 100.0, w)
            want[i] = np.where(on, w, 0.0)
        top = k1z[m] == 2   # columns whose surface is in the first layer: no dry layers to fold in
        assert top.sum() > 1000
        np.testing.assert_array_equal(wp[:, m][:, top], want[:, top])
    finally:
        g.close()
