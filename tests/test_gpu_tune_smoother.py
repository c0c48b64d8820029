"""bcg_autotune(SMOOTHER) times the smoother form that its choice steers, on levels
that an FP64 solve takes in another form too (register tiles, which have no
target), and the FP64 solve keeps those."""
import pytest

from baccolonygrowth_b200 import params
from baccolonygrowth_b200.colony import Colony, workload_colony


def kernels(torch, call):
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        call()
        torch.cuda.synchronize()
    return [e.name for e in prof.events()]


@pytest.mark.gpu
def test_tuner_times_the_form_it_steers(gpu):
    import torch
    torch.zeros(1, device="cuda")
    col = Colony(params.workload_params("scale_262k"), workload_colony("scale_262k", n=20000))
    col.update_density()
    col.deplete_wall()
    seen = kernels(torch, lambda: col.mg_solve(1))
    if not any("k_mg" in k for k in seen):
        pytest.skip("the profiler records no kernels here")
    assert any("k_mg_tile" in k for k in seen) and not any("k_mg_smooth_tma" in k for k in seen)
    seen = kernels(torch, lambda: col.autotune("SMOOTHER"))
    assert sum("k_mg_smooth_tma" in k for k in seen) == 9 * 4 and not any("k_mg_tile" in k for k in seen)
    assert any("k_mg_tile" in k for k in kernels(torch, lambda: col.mg_solve(1)))
    col.close()
