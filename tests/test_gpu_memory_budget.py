"""Device memory of the blocked self-energy: what a call allocates beyond its fixed buffers stays within the budget that
the caller set, digit planes included."""
import gc

import numpy as np
import pytest

from gb200 import lib, solvers, synth

pytestmark = pytest.mark.gpu


def _free():
    import torch
    gc.collect()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info(0)[0]


def _footprint(s, slices, budget):
    """(bytes that one self-energy call allocates, the self-energy)"""
    with solvers.make_context(s, precision=lib.PREC_SPLIT if slices else lib.PREC_FP64, slices=slices or 4) as c:
        c.set_memory_budget(budget)
        before = _free()
        out = c.gw_sigma(s.G)
        return before - _free(), out


@pytest.mark.parametrize("ns,nao,naux,slices", [(1, 16, 96, 5), (2, 16, 96, 6), (1, 6, 40, 5), (1, 16, 96, 8), (1, 16, 96, 0)])
def test_blocks_and_planes_stay_within_the_budget(gpu, ns, nao, naux, slices):
    # (nao = 6: the digits of a 6-long contraction are padded to 64 bytes, which makes T1's planes the largest)
    s = synth.make_system(mesh=(4, 2, 2), nao=nao, naux=naux, ns=ns, beta=20.0, nts=60, eps_range=2.0, seed=2)
    x1 = 16.0 * 60 * ns * naux * nao * nao  # one intermediate of one k-point
    _footprint(s, slices, 1.0)              # (loads the kernels)
    single, ref = _footprint(s, slices, 1.0)  # blocks of one k-point, with the fixed buffers
    for blocks in (12.0, 24.0):
        budget = blocks * x1
        got, out = _footprint(s, slices, budget)
        # (`single` holds a block too: room for the granules of a few dozen allocations)
        assert got - single <= budget
        assert np.abs(out - ref).max() <= 1e-8 * np.abs(ref).max()
