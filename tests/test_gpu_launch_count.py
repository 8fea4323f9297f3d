"""The library's count of its kernel launches (gb200_stats_read) against what the CUDA profiler sees, for a self-energy
whose contractions take the slicers' one-pass, resident and two-pass forms."""
import pytest

from gb200 import lib, solvers, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("slices", [0, 5])
def test_launch_count_matches_the_profiler(gpu, slices):
    import torch
    from torch.profiler import ProfilerActivity, profile
    s = synth.make_system(mesh=(2, 1, 1), nao=16, naux=100, ns=1, beta=10.0, nts=14, eps_range=1.0, seed=1)
    with solvers.make_context(s, precision=lib.PREC_SPLIT if slices else lib.PREC_FP64, slices=slices or 4) as c:
        c.gw_sigma(s.G)
        torch.cuda.synchronize()
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            before = c.stats_read()[0]
            c.gw_sigma(s.G)
            torch.cuda.synchronize()
            counted = c.stats_read()[0] - before
    kernels = [e for e in prof.events() if e.device_type == torch.autograd.DeviceType.CUDA and not e.name.startswith(("Memcpy", "Memset"))]
    if not kernels:
        pytest.skip("the CUDA profiler reports nothing here (another tool may hold it)")
    assert counted == len(kernels), sorted({e.name for e in kernels})
