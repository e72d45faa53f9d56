"""The multigrid solve on both sides of the size where level 1's red half-sweep of the way up becomes
a phase of its own: level 0 in one pass of the grid's threads (75,520 groups of four cells for
75,776 threads on 148 SMs) and just more (76,800).  Against the FP64 loop: both stop at a relative residual of 1e-12
(|b| below 1e3, smallest eigenvalue at least 1), and two steps of three solves feed on each other."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(640, 472), (640, 480)])
def test_multigrid_against_fp64(native_libs, tmp_path, nx, ny):
    from si3d_b200 import native, synth
    from si3d_b200.model import GpuRun
    rng = np.random.default_rng(ny)
    depth = np.round(rng.uniform(1.0, 3.0, (nx, ny)), 1)
    u = 4.0 + rng.uniform(-1.0, 1.0, (nx, ny))
    d = str(tmp_path / "lake")
    synth.write_run(synth.Basin("lake", nx, ny, 100.0, 100.0, depth, 3, 1.0, 20.0, 100, dzmin=0.1, uair=u, vair=0.0 * u), d)
    out = {}
    for name in ("FP64", "MIXED_MG"):
        g = GpuRun(d, pcg_itmax=4000, precision=getattr(native, f"SI3D_{name}"))
        try:
            st = g.run(2)
            assert all(s.ier[i] == 0 for s in st for i in range(s.nsolves))
            out[name] = g.get("s")
        finally:
            g.close()
    assert np.abs(out["FP64"]).max() > 1e-6
    assert np.abs(out["MIXED_MG"] - out["FP64"]).max() <= 1e-9
