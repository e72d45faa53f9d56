"""Surface layers that dry and rewet: a shallow lake of thin layers under a wind that lowers its upwind
side by more than a layer.  Covers the branches for a dried surface layer in the surface-layer stage and
its short form inside fd, the velocities (transport of a dried layer to the one below), both continuity
forms (the dry layers' fluxes folded into the surface layer) and the momentum kernels."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_fd_paths import FIELDS, OTHER
from test_gpu_parity import STATE_2D, STATE_3D, STATE_I, _cmp, _pair

pytestmark = pytest.mark.gpu


def lake(path, nx, ny, ddz, dmin, dmax):
    from si3d_b200 import synth
    f = synth.gaussian_field((nx, ny), 3.0, np.random.default_rng(1))
    depth = np.round((dmin + (dmax - dmin) * (f - f.min()) / (f.max() - f.min())) * 10) / 10
    u = np.full((nx, ny), float(synth.wind_speed_for_stress(0.2)))
    b = synth.Basin("dry", nx, ny, 100.0, 100.0, depth, int(np.ceil(dmax / ddz - 1e-9)), ddz, 20.0, 1000, dzmin=0.01,
                    uair=u, vair=0.3 * u, t_top=20.0, t_bottom=15.0)
    synth.write_run(b, str(path))
    return str(path)


# layers of 3 cm over 0.1 to 0.6 m (columns of 4 to 20), of 5 cm over 0.1 to 0.4 m (2 to 8)
@pytest.fixture(scope="module", params=[(24, 16, 0.03, 0.1, 0.6, 40), (17, 29, 0.05, 0.1, 0.4, 30)], ids=["3cm", "5cm"])
def dry(request, tmp_path_factory):
    *shape, steps = request.param
    return lake(tmp_path_factory.mktemp("dry"), *shape), steps


def surfaces(run):
    return [run.get(k).copy() for k in STATE_I]


@pytest.mark.parametrize("more", [0, 60])   # later some layers are wet again
def test_fd_ends_as_its_stages_do(native_libs, dry, more):
    """Twelve time steps of fd calls against the stage calls, bit for bit, while layers dry and rewet."""
    from si3d_b200 import native
    from si3d_b200.model import GpuRun
    path, steps = dry[0], dry[1] + more
    a, b = GpuRun(path, pcg_itmax=2000), GpuRun(path, pcg_itmax=2000)
    try:
        a.run(steps)
        b.run(steps)
        down, up = np.zeros(3, int), np.zeros(3, int)

        def fd(n, istep, last):
            before = surfaces(a)
            native.check(a.g.si3d_gpu_fd(a.gh, n, istep, last, C.byref(native.StepStats())))
            for s in ("momentum", "matcon", "solve", "vel", "scalar", "vel2"):
                b.stage(s, istep)
            for f in FIELDS + OTHER + list(STATE_I):
                np.testing.assert_array_equal(a.get(f), b.get(f), err_msg=f"{f}, step {n}, {istep}")
            for q, (x, y) in enumerate(zip(before, surfaces(a))):
                down[q] += (y > x).sum()

        for n in range(steps + 1, steps + 13):
            tops = surfaces(a)
            fd(n, 1, 0)
            for r in (a, b):
                native.check(r.g.si3d_gpu_settrap(r.gh))
            fd(n, 2, 0)
            for r in (a, b):
                native.check(r.g.si3d_gpu_settrap2(r.gh))
            fd(n, 2, 1)
            for r in (a, b):
                native.check(r.g.si3d_gpu_save(r.gh, 2))
            for q, (x, y) in enumerate(zip(tops, surfaces(a))):
                up[q] += (y < x).sum()
        assert (down > 0).all() if more == 0 else down.sum() > 0 and up.sum() > 0
    finally:
        a.close()
        b.close()


@pytest.mark.parametrize("istep", [1, 2])
def test_stages_against_the_oracle(native_libs, oracle_lib, dry, istep):
    """Each stage from the oracle's state, tolerances as for the basin that stays wet.  (Not the momentum
    stage: at a face with a dry cell the oracle leaves the layers below it to the call before.)"""
    path, steps = dry
    o, g = _pair(path, oracle_lib, steps=steps)
    try:
        assert (o.geti("k1z")[:-1] > 2).sum() > 20
        for stage, fields, tol in [("momentum", [], 0.0),
                                   ("matcon", ["sx", "sy", "dd", "qq", "rr"], 1e-14),
                                   ("solve", ["s", "h", "hu", "hv"], 1e-11),
                                   ("vel", ["uh", "vh", "wp", "k1z", "k1u", "k1v"], 1e-9),
                                   ("scalar", ["sal", "Bth2", "Bth3", "Bth4"], 1e-9),
                                   ("vel2", ["h", "hu", "hv", "uh", "vh"], 1e-9)]:
            o.stage(stage, istep)
            g.stage(stage, istep)
            _cmp(o, g, fields, tol, f"{stage}/istep{istep}")
            for f in STATE_3D + STATE_2D:
                g.set(f, o.get(f))
            for f in STATE_I:
                g.set(f, o.geti(f))
    finally:
        g.close()


def test_fused_momentum_kernel_is_bit_identical(native_libs, dry):
    from si3d_b200.model import GpuRun
    path, steps = dry
    state = {}
    for lanes in (8, 1):
        g = GpuRun(path, pcg_itmax=2000)
        try:
            g.set_tune((lanes, 128, 8, 128))
            g.run(steps + 10)
            state[lanes] = {f: g.get(f).copy() for f in FIELDS + OTHER}
        finally:
            g.close()
    for f, want in state[8].items():
        np.testing.assert_array_equal(state[1][f], want, err_msg=f)


@pytest.fixture(scope="module")
def wide(tmp_path_factory):
    """More than 65536 columns, of which the upwind ones have dried layers: one thread per column."""
    return lake(tmp_path_factory.mktemp("wide"), 270, 250, 0.03, 0.1, 0.6)


def test_continuity_folds_the_dry_layers(native_libs, wide):
    """wp against the layer sums of the same state, the dry layers' added to the surface layer's, in
    continuity(2)'s order."""
    from si3d_b200.model import GpuRun
    g = GpuRun(wide, pcg_itmax=4000)
    try:
        assert g.lm >= 65536
        g.run(60)
        uhp, vhp, wp, k1z, kmz = g.get("uhp"), g.get("vhp"), g.get("wp"), g.get("k1z"), g.map("kmz")
        lW, lS = g.map("lWC"), g.map("lSC")
        m = np.arange(g.lm)
        x = (uhp[:, m] - uhp[:, lW[m] - 1]) / 100.0
        y = (vhp[:, m] - vhp[:, lS[m] - 1]) / 100.0
        w, want = np.zeros(g.lm), np.zeros((g.km1, g.lm))
        for k in range(g.km1, 1, -1):
            on = (k <= kmz[m]) & (k >= k1z[m])
            w = np.where(on, w - x[k - 1] - y[k - 1], w)
            want[k - 1] = np.where(on, w, 0.0)
        folded = np.zeros(g.lm, bool)
        for k in range(2, int(k1z[m].max())):
            on = (k < k1z[m]) & (k1z[m] <= kmz[m])
            w = np.where(on, w - x[k - 1] - y[k - 1], w)
            folded |= on & ((x[k - 1] != 0) | (y[k - 1] != 0))
        wet = k1z[m] <= kmz[m]
        want[k1z[m][wet] - 1, m[wet]] = w[wet]
        assert folded.sum() > 100
        np.testing.assert_array_equal(wp[:, m][:, wet], want[:, wet])
    finally:
        g.close()


def test_velocity_stage_of_many_columns_against_the_oracle(native_libs, oracle_lib, wide):
    """Velocities and continuity(1) with one thread per column, from the device's state."""
    from si3d_b200.model import GpuRun
    g = GpuRun(wide, pcg_itmax=4000)
    try:
        g.run(60)
        for s in ("momentum", "matcon", "solve"):
            g.stage(s, 1)
        o = oracle_lib.OracleRun(wide, ordering=1, pcg_itmax=4000)
        for f in STATE_3D + STATE_2D:
            o.set(f, g.get(f))
        for f in STATE_I:
            o.seti(f, g.get(f))
        before = g.get("k1u").copy()
        o.stage("vel", 1)
        g.stage("vel", 1)
        assert (g.get("k1u") > before).sum() > 0 and (g.get("k1z")[:-1] > 2).sum() > 100
        _cmp(o, g, ["uh", "vh", "wp", "k1z", "k1u", "k1v"], 1e-12, "vel")
    finally:
        g.close()
