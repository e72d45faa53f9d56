"""The handle's count of launched kernels."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lanes,momentum", [(1, 5), (8, 7)])
def test_kernels_of_an_fd_call(native_libs, run_dirs, lanes, momentum):
    """Density sums, and for each direction the fused or the cell and column kernels and the back
    substitution; zeta assembly 1, solve set-up 7, loop 1, end 2, surface layer 1, velocities and
    continuity 3, temperature 3, layers 1."""
    from si3d_b200 import native
    from si3d_b200.model import GpuRun
    run = GpuRun(run_dirs["t1"], pcg_itmax=2000)
    try:
        run.set_tune((lanes, 128, 8, 128))
        run.run(2)
        before, _ = run.counters()
        native.check(run.g.si3d_gpu_fd(run.gh, 3, 1, 0, C.byref(native.StepStats())))
        after, _ = run.counters()
        assert after - before == momentum + 19
    finally:
        run.close()
