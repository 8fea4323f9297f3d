"""The allocation-free Fock build at sizes that take different tile variants of the FP64 GEMM: after one first call in
the context, calls of other sizes leave the free device memory as it is, also while the stream is captured into a graph,
and give the Fock matrix of the allocating entry point (sums in the same order: equal to 1e-13 of its largest element)."""
import numpy as np
import pytest

from gb200 import lib, synth

pytestmark = pytest.mark.gpu


def _run(s, V, dm, S, F, stream):
    lib.hf_fock_noalloc(s.nk, s.nao, s.ns, s.NQ, V.data_ptr(), dm.data_ptr(), S.data_ptr(), 0.2, F.data_ptr(), stream)


def _inputs(nao, naux, ns):
    import torch
    s = synth.make_system(mesh=(2, 1, 1), nao=nao, naux=naux, ns=ns, beta=10.0, nts=14, eps_range=1.0, seed=nao)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    return s, t(s.V_full()), t((-1.0 if ns == 2 else -2.0) * s.G[-1]), t(s.S)


def test_other_sizes_after_the_first_call(gpu):
    import torch
    from gb200 import solvers
    s, V, dm, S = _inputs(6, 20, 1)
    _run(s, V, dm, S, torch.empty_like(dm), 1)
    torch.cuda.synchronize()
    for nao, naux, ns in ((5, 13, 2), (17, 40, 1), (33, 70, 1), (40, 64, 2)):
        s, V, dm, S = _inputs(nao, naux, ns)
        F, Fc = torch.empty_like(dm), torch.zeros_like(dm)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        _run(s, V, dm, S, F, 1)
        torch.cuda.synchronize()
        assert torch.cuda.mem_get_info()[0] == free
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            _run(s, V, dm, S, Fc, torch.cuda.current_stream().cuda_stream)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(F, Fc)
        with solvers.make_context(s) as c:
            want = c.hf_fock(dm.cpu().numpy(), s.S, 0.2)
        assert np.abs(F.cpu().numpy() - want).max() <= 1e-13 * np.abs(want).max()
