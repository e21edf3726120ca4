"""The pinned words a solve's steps report their residuals in: contexts that solve
batches of different widths one after another (kept blocks, blocks too wide to be
kept), a column at a time and several thousand.

A solved column has an explicit residual ||b - A x|| below the tolerance by the
solver's own test.  The oracle's operator gives the same residual up to rounding of
the order of 1e-15 ||A|| ||x||, below 1e-10 ||b|| for ||A|| ||x|| up to 1e5 ||b||:
1e-4 of the tolerance, which is 1e-6 ||b||.
"""
import numpy as np
import pytest

from oracle import keywords, model
from plasmonx_b200 import configs
from plasmonx_b200.inputs import Problem
from plasmonx_b200.solver import Context, Solver

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def ctx():
    c = Context(0)
    yield c
    c.close()


@pytest.mark.parametrize('n_freq', [1, 85, 86, 1400, 2])
@pytest.mark.parametrize('precision', ['fp64', 'mixed_bf16x3'])
def test_batches_of_many_widths_in_one_context(ctx, n_freq, precision):
    """Two words a column and three columns a frequency: 510 words fill the smallest block,
    8,400 are past the largest kept one."""
    text = configs.na_sphere(radius=9.0, n_freq=n_freq, method='iterative').to_keyword_text()
    p, s = Problem.from_keyword_text(text), model.System.from_keywords(keywords.read_keyword_text(text))
    op = model.Operator(s)
    tol = 1e-6 * np.linalg.norm(op.rhs(0)[:, 0])
    with Solver(p, ctx=ctx, store_t=True) as sv:
        out = sv.solve(precision=precision, tol=tol, max_krylov=p.n_var, want_x=True)
    assert (out['status'] == 0).all()
    for f in sorted({0, n_freq // 2, n_freq - 1}):
        b = op.rhs(f)
        for pol in range(b.shape[1]):
            assert np.linalg.norm(b[:, pol] - op.matvec(f, out['x'][f, :, pol])) <= tol * (1.0 + 1e-4)
