"""Shifted Hessenberg direct solve at the orders where its kernels change path:
the smallest orders, edges of the 64-row and 32-column tiles and of the 32-unknown
blocks of the back substitution, orders whose tiles are doubled (above 896) and
whose rows exceed what a thread loads ahead (above 2,048).

Against the oracle's matrix: the backward error ||b - A x|| / (||A||_F ||x|| + ||b||)
of a backward-stable solve is at most a small multiple of n eps; held to
(10 + n) eps, and the columns of a grid to those of a single frequency bit for bit
within one contraction kernel.
"""
import numpy as np
import pytest

from oracle import keywords, model
from plasmonx_b200 import configs, geometry
from plasmonx_b200.inputs import Problem
from plasmonx_b200.solver import Context, Solver

pytestmark = pytest.mark.gpu

EPS = 2.220446049250313e-16


@pytest.fixture(scope='module')
def ctx():
    c = Context(0)
    yield c
    c.close()


def _sodium(n, n_freq):
    pts = geometry.sphere('bcc', 4.225, 30.0, 0.01, 1)
    pts = pts[np.argsort((pts ** 2).sum(1), kind='stable')][:n]
    p0 = configs.build('wfq', pts, ['Na'], np.zeros(n, np.int32), configs.ev_grid(2.0, 4.0, n_freq),
                       method='inversion')
    text = p0.to_keyword_text()
    return Problem.from_keyword_text(text), model.System.from_keywords(keywords.read_keyword_text(text))


@pytest.mark.parametrize('n', [3, 4, 5, 31, 32, 33, 34, 63, 64, 65, 66, 127, 160, 896, 900, 1030, 2049, 2100])
def test_backward_error(ctx, n):
    n_freq = 3 if n < 2000 else 1
    p, s = _sodium(n, n_freq)
    op = model.Operator(s)
    with Solver(p, ctx=ctx, store_t=True) as sv:
        out = sv.solve(mode='inversion', want_x=True)
        b = np.stack([sv.rhs(i, 7) for i in range(n_freq)])
    assert (out['status'] == 0).all()
    for i in range(n_freq):
        A, x = op.matrix(i), out['x'][i]
        r = np.linalg.norm(b[i] - A @ x, axis=0)
        bar = (10 + n) * EPS * (np.linalg.norm(A) * np.linalg.norm(x, axis=0) + np.linalg.norm(b[i], axis=0))
        assert np.all(r <= bar), r / bar


def test_budget_too_small_for_the_reduction_falls_back(ctx):
    """A context whose budget holds the LU's matrix but not the reduction's still solves."""
    p, s = _sodium(600, 2)
    with Solver(p, ctx=ctx, store_t=True) as sv:
        ref = sv.solve(mode='inversion')
    n2 = 8 * 600 * 600
    small = Context(0, hbm_budget=5 * n2)
    try:
        with Solver(p, ctx=small, store_t=True) as sv:
            out = sv.solve(mode='inversion')
    finally:
        small.close()
    assert (out['status'] == 0).all()
    assert np.max(np.abs(out['results'] - ref['results'])) <= 1e-10 * np.abs(ref['results']).max()
