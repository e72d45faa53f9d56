"""The fused momentum kernel's tiles at their edges: basins smaller than a tile, one row or one column
wide, a grid that fills tiles exactly, and scattered land, where a tile's columns run out before its
faces do.  Against the split cell + column kernels, which evaluate the same expressions in the same
order: the results are the same, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def lake(nx, ny, land, layers, seed):
    from si3d_b200 import synth
    rng = np.random.default_rng(seed)
    depth = np.round(rng.uniform(1.5, layers, (nx, ny)), 1)
    depth[rng.random((nx, ny)) < land] = -9.9
    depth[nx // 2, ny // 2] = float(layers)
    u = np.full((nx, ny), 4.0) + rng.uniform(-1.0, 1.0, (nx, ny))
    return synth.Basin("lake", nx, ny, 100.0, 100.0, depth, layers, 1.0, 20.0, 100, dzmin=0.1, uair=u, vair=0.3 * u)


@pytest.mark.parametrize("nx,ny,land,layers", [(3, 2, 0.0, 4), (40, 1, 0.0, 6), (1, 40, 0.0, 6), (16, 32, 0.0, 9),
                                               (33, 65, 0.0, 5), (48, 70, 0.35, 12), (60, 40, 0.6, 3)])
def test_fused_and_split_momentum_agree(native_libs, tmp_path, nx, ny, land, layers):
    from si3d_b200 import synth
    from si3d_b200.model import GpuRun
    d = str(tmp_path / "lake")
    synth.write_run(lake(nx, ny, land, layers, nx * 100 + ny), d)
    names = ("s", "uh", "vh", "agx", "arx", "agy", "ary", "eagx", "earx", "eagy", "eary")
    got = {}
    for lanes in (8, 1):
        g = GpuRun(d, pcg_itmax=4000)
        try:
            g.set_tune((lanes, 128, 8, 128))
            g.run(4)
            got[lanes] = {n: g.get(n).copy() for n in names}
        finally:
            g.close()
    for n in names:
        np.testing.assert_array_equal(got[1][n], got[8][n], err_msg=n)
    assert np.isfinite(got[1]["s"]).all()
