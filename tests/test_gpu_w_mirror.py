"""Split-precision self-energies on grids on both sides of the rule that takes W through its mirror-symmetric form: a
Chebyshev grid whose matrices are symmetric only to their round-off, and the same grid made asymmetric, which must be
applied as given.  Against the FP64 path, which always applies the matrices as given.

Tolerance: five base-256 slices hold 39 bits.  The relative error of these self-energies is 1e-11 at the workload's
sizes; five base-128 slices (35 bits) keep 9e-10 over the measured range, and four bits more give 5.6e-11."""
import copy
import dataclasses

import numpy as np
import pytest

from gb200 import lib, solvers, synth

pytestmark = pytest.mark.gpu
TOL = 9e-10 / 16


def sigma(s, slices):
    with solvers.make_context(s, precision=lib.PREC_SPLIT if slices else lib.PREC_FP64, slices=slices or 4) as c:
        return c.gw_sigma(s.G)


@pytest.mark.parametrize("ns", [1, 2])
def test_grid_symmetric_to_round_off(gpu, ns):
    s = synth.make_system(mesh=(2, 1, 1), nao=6, naux=22, ns=ns, beta=200.0, nts=118, eps_range=5.0, seed=4)
    ref = sigma(s, 0)
    assert np.linalg.norm(sigma(s, 5) - ref) <= TOL * np.linalg.norm(ref)


@pytest.mark.parametrize("ns", [1, 2])
def test_asymmetric_grid_is_applied_as_given(gpu, ns):
    s = synth.make_system(mesh=(2, 1, 1), nao=6, naux=22, ns=ns, beta=20.0, nts=24, eps_range=2.0, seed=3)
    plain = sigma(s, 5)
    g = copy.copy(s.grid)
    g.Ttn_b = g.Ttn_b.copy()
    g.Ttn_b[12:] *= 1 + 1e-6
    t = dataclasses.replace(s, grid=g)
    ref = sigma(t, 0)
    got = sigma(t, 5)
    assert np.linalg.norm(got - ref) <= TOL * np.linalg.norm(ref)
    assert np.linalg.norm(got - plain) >= 1e3 * TOL * np.linalg.norm(ref)  # what mirroring would have lost shows
