"""Screened interaction where I - P(i Omega) is not positive definite: the block inverse flags such a matrix and the
pivoted Gauss-Jordan kernels invert it from the untouched input, beside matrices of the same batch that stay with the
block inverse.  A Green's function multiplied by i a turns the sign of the polarization, so its large eigenvalues pass 1
at low frequencies and not at high ones.  Sizes around the splits into leaves of 64, and one whose panel does not fit the
blocked kernel's shared memory; against the oracle."""
import numpy as np
import pytest

import gw_oracle as O
from gb200 import lib, solvers, synth

pytestmark = pytest.mark.gpu


def spectra(s, G):
    """Eigenvalues of I - P(i Omega) [nk][nw_b][NQ] (lower triangle and real diagonal, as the solve reads it)."""
    V, bz = O.HalfStoredIntegrals(s.V_half), O.NoSymBZ(s.mesh)
    out = []
    for q in range(s.nk):
        P0 = np.zeros((s.nts, s.NQ, s.NQ), dtype=complex)
        for k in range(s.nk):
            kq = bz.k1_from_k2q(k, q)
            O.eval_P0_tilde(G, V.pair(k, kq), k, kq, P0, s.ns)
        O.symmetrize_P0(P0, s.nk)
        Pw = np.tensordot(s.grid.Tnt_b, P0, 1)
        out.append([np.linalg.eigvalsh(np.eye(s.NQ) - O.hermitian_from_lower(p)) for p in Pw])
    return np.array(out)


@pytest.mark.parametrize("naux,mesh", [(65, (2, 1, 1)), (127, (2, 1, 1)), (129, (2, 1, 1)), (193, (1, 1, 1)), (720, (1, 1, 1))])
def test_indefinite_and_definite_matrices_of_one_batch(gpu, naux, mesh):
    s = synth.make_system(mesh=mesh, nao=4, naux=naux, ns=1, beta=10.0, nts=14, eps_range=1.0, seed=naux)
    w = 1.0 - spectra(s, s.G)  # eigenvalues of P; those of -a^2 P below

    def conditioned(a):
        e = 1.0 + a * a * w
        bad = np.mean(e.min(axis=2) < 0)
        return np.abs(e).max() / np.abs(e).min() if 0.2 <= bad <= 0.8 else np.inf

    a = min(np.geomspace(0.3, 30.0, 400), key=conditioned)
    G = 1j * a * s.G
    e = spectra(s, G)
    bad = (e.min(axis=2) < 0).ravel()
    assert bad.any() and not bad.all()
    cond = np.abs(e).max() / np.abs(e).min()
    assert cond < 1e4
    ref = O.gw_solve(G, O.HalfStoredIntegrals(s.V_half), O.NoSymBZ(s.mesh), s.grid.Tnt_b, s.grid.Ttn_b, s.ns, s.NQ)
    with solvers.make_context(s, precision=lib.PREC_FP64) as c:
        got = c.gw_sigma(G)
    # two backward stable inverses differ by about n eps cond
    tol = max(1e-12, naux * 2.3e-16 * cond)
    assert np.abs(got - ref).max() <= tol * np.abs(ref).max()
