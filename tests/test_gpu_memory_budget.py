"""Device memory of the blocked self-energy: what a call allocates beyond its fixed buffers stays within the budget that
the caller set, digit planes included, and without a budget the buffers of one call do not make the next one choose
smaller blocks."""
import gc

import numpy as np
import pytest

from gb200 import batch, lib, solvers, synth

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


@pytest.mark.parametrize("slices", [0, 5])
def test_a_second_call_takes_the_same_blocks(gpu, slices):
    """With memory for about half of the k-points: the same launches and the same bits, call after call."""
    import torch
    s = synth.make_system(mesh=(4, 2, 2), nao=24, naux=140, ns=1, beta=20.0, nts=80, eps_range=2.0, seed=1)
    per_k = 16.0 * 80 * 140 * 24 * 24 * (2.75 if slices else 2.0)
    with solvers.make_context(s, precision=lib.PREC_SPLIT if slices else lib.PREC_FP64, slices=slices or 4) as c:
        c.set_memory_budget(1.0)
        c.gw_sigma(s.G)  # the kernels and the buffers of fixed size
        c.set_memory_budget(0.0)
        ballast = torch.empty(int(_free() - 8 * per_k / 0.6), dtype=torch.uint8, device="cuda")
        try:
            out, launches = [], []
            for _ in range(3):
                before = c.stats_read()[0]
                out.append(c.gw_sigma(s.G))
                launches.append(c.stats_read()[0] - before)
        finally:
            del ballast
            torch.cuda.empty_cache()
    assert launches[0] == launches[1] == launches[2]
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])


def test_contexts_of_one_batched_call_share_what_is_free(gpu):
    """Four systems whose blocks would each take most of the free memory, without budgets: together they fit."""
    import torch
    systems = [synth.make_system(mesh=(4, 2, 2), nao=24, naux=140, ns=1, beta=20.0, nts=80, eps_range=2.0, seed=i) for i in range(4)]
    per_k = 16.0 * 80 * 140 * 24 * 24 * 2.75
    ctxs = [solvers.make_context(s, precision=lib.PREC_SPLIT, slices=5) for s in systems]
    try:
        b = batch.SystemBatch(ctxs)
        G = [torch.from_numpy(s.G).cuda() for s in systems]
        Sig = [torch.empty_like(g) for g in G]
        gp, sp = [x.data_ptr() for x in G], [x.data_ptr() for x in Sig]
        with solvers.make_context(systems[0], precision=lib.PREC_SPLIT, slices=5) as c:
            c.set_memory_budget(1.0)
            before = _free()
            ref = c.gw_sigma(systems[0].G)
            single = before - _free()  # one context's fixed buffers and a block of one k-point
        ballast = torch.empty(int(_free() - 12 * per_k - 4 * single), dtype=torch.uint8, device="cuda")
        try:
            b.run_gw_grouped(gp, sp)
            torch.cuda.synchronize()
        finally:
            del ballast
            torch.cuda.empty_cache()
        assert np.abs(Sig[0].cpu().numpy() - ref).max() <= 1e-8 * np.abs(ref).max()
    finally:
        for c in ctxs:
            c.close()
