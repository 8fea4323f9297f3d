"""Edges of the split contraction kernel's tiles: the tensor-core engine against the CUDA-core validation engine, bit for
bit, on systems whose contractions have fewer rows than a tile, remainders of rows, columns and K steps, one and two
accumulator sets (short contractions run with two for up to five slices), one time or a mirror pair per screened
interaction, and a column width set by the caller."""
import numpy as np
import pytest

from gb200 import lib, solvers, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nao,naux,ns,slices,width", [(3, 5, 1, 5, 0), (17, 61, 2, 5, 0), (16, 64, 1, 4, 32),
                                                      (33, 70, 1, 6, 0), (40, 130, 1, 5, 16), (12, 129, 2, 2, 0),
                                                      (9, 40, 1, 8, 0)])
def test_engines_agree_bit_for_bit(gpu, nao, naux, ns, slices, width):
    s = synth.make_system(mesh=(2, 1, 1), nao=nao, naux=naux, ns=ns, beta=10.0, nts=14, eps_range=1.0, seed=nao)
    out = []
    for engine in (0, 1):
        with solvers.make_context(s, precision=lib.PREC_SPLIT, slices=slices) as c:
            c.set_split_engine(engine)
            c.set_tile_width(width)
            out.append(c.gw_sigma(s.G))
    assert np.isfinite(out[0]).all()
    assert np.array_equal(out[0], out[1])
