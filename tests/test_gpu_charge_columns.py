"""Charge rows with columns across the lanes (many columns, one atom type) against the
rows' own form (few columns): the same sums in the same order, so the same bits.  Column
counts around the switch (12) and the tiles of 32; rows shorter than a tile of 32
entries, and up to 530 entries (past the 512 that the row form keeps in registers).
"""
import numpy as np
import pytest

from plasmonx_b200 import configs
from plasmonx_b200.solver import Context, Solver

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def ctx():
    c = Context(0)
    yield c
    c.close()


@pytest.mark.parametrize('shape, radius', [('na', 5.0), ('na', 9.0), ('na', 20.0), ('ag', 9.0)])
@pytest.mark.parametrize('n_freq', [11, 12, 13, 31, 33, 65])
def test_columns_have_the_bits_of_small_batches(ctx, shape, radius, n_freq):
    make = configs.na_sphere if shape == 'na' else configs.ag_sphere
    p = make(radius=radius, n_freq=n_freq, method='iterative')
    with Solver(p, ctx=ctx, store_t=True) as sv:
        kw = dict(precision='fp64', pol_mask=1, tol=1e-30, max_krylov=3, want_x=True, trace=True)
        a, b = sv.solve(**kw), sv.solve(freq_block=4, **kw)
    assert np.isfinite(a['trace'][:, 0]).all() and (a['trace'][:, 0, 0] > 0).all()
    np.testing.assert_array_equal(a['trace'], b['trace'])
    np.testing.assert_array_equal(a['x'], b['x'])
