"""An ensemble in which one member is too small for the loop on the black unknowns: the others' solves
stay batched, the pond solves beside them, and each gives what it gives alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_a_pond_leaves_the_others_batched(native_libs, tmp_path):
    from si3d_b200 import ensemble, native, synth
    from si3d_b200.ensemble import Ensemble
    from si3d_b200.model import GpuRun
    members = ensemble.basins(n=2, seed=12, size_min=(30, 20), size_max=(90, 60), layers=(6, 14))
    depth = np.full((6, 5), 4.0)
    depth[0, 0] = depth[5, 4] = 0.0   # 28 columns, 14 of a colour
    wind = float(synth.wind_speed_for_stress(0.1))
    members.insert(1, synth.Basin("pond", 6, 5, 50.0, 50.0, depth, 5, 1.0, members[0].dt, 100, dzmin=0.1,
                                  uair=np.full((6, 5), wind), vair=np.zeros((6, 5))))
    dirs = ensemble.write(members, str(tmp_path))
    steps = 5
    ens = Ensemble(dirs)
    try:
        iters, ier, _ = ens.step(steps)
        assert (ier == 0).all()
        assert ens.solve_blocks() > 0
        got = [{f: r.get(f).copy() for f in ("s", "uh", "sal")} for r in ens.runs]
        ens.solve_mode(native.SI3D_ENS_SOLVE_MEMBERS)
        ens.step(1)
        assert ens.solve_blocks() == 0
        ens.solve_mode(native.SI3D_ENS_SOLVE_BATCHED)
        ens.step(1)
        assert ens.solve_blocks() > 0
        end = [r.get("s").copy() for r in ens.runs]
    finally:
        ens.close()
    for k, d in enumerate(dirs):
        run = GpuRun(d, pcg_itmax=2000)
        try:
            st = run.run(steps)
            for f, want in got[k].items():
                np.testing.assert_array_equal(run.get(f), want, err_msg=f)
            for s in range(1, steps):
                ref = [st[s].iters[i] for i in range(st[s].nsolves)]
                assert list(iters[s, k, :len(ref)]) == ref
            run.run(2)
            np.testing.assert_array_equal(run.get("s"), end[k])
        finally:
            run.close()
