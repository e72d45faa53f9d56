"""Device memory that a handle takes."""
import pytest

pytestmark = pytest.mark.gpu


def test_a_small_basin_takes_little_memory(native_libs, run_dirs):
    """Twenty handles of a basin whose arrays come to less than 2 MB: at most 8 MB each (slabs of 32 MB
    took four times that)."""
    import torch
    from si3d_b200.model import GpuRun
    first = GpuRun(run_dirs["t0"])   # the context and the kernels' code are loaded
    try:
        assert first.lm * first.km1 * 8 * 40 < 2 << 20
        before = torch.cuda.mem_get_info()[0]
        runs = [GpuRun(run_dirs["t0"]) for _ in range(20)]
        taken = before - torch.cuda.mem_get_info()[0]
        for r in runs:
            r.close()
        assert taken <= 20 * (8 << 20)
    finally:
        first.close()
