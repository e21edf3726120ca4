"""Arnoldi step of the batched GMRES at the sizes where its kernels change path:
tile edges of the Givens chain and the back substitution (32), the switch from
modified to classical Gram-Schmidt (25), the first steps.

After m steps the returned x is the least-squares solution over m basis
vectors, so the explicit residual ||b - A x|| (the oracle's operator) equals the
recurrence's residual |g_{m+1}|.  The two differ by rounding of the order of
1e-15 ||A|| ||x|| against a residual of at least 1e-6 ||b||: held to 1e-6 of the
residual.
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


@pytest.mark.parametrize('steps', [1, 2, 24, 25, 26, 31, 32, 33, 34, 64, 65, 66])
def test_residual_after_a_given_number_of_steps(ctx, steps):
    p0 = configs.ag_sphere(radius=8.0, n_freq=2, method='iterative')
    text = p0.to_keyword_text()
    p, s = Problem.from_keyword_text(text), model.System.from_keywords(keywords.read_keyword_text(text))
    op = model.Operator(s)
    rng = np.random.default_rng(steps)
    b = rng.standard_normal(p.n_var) + 1j * rng.standard_normal(p.n_var)
    with Solver(p, ctx=ctx, store_t=True) as sv:
        _, n, trace = sv.gmres(1, b, tol=1e-5 * np.linalg.norm(b), restart=p.n_var)
        assert n > 66
        # the residuals of GMRES do not increase: this tolerance is first met after `steps` steps
        tol = trace[steps - 1] * (1.0 + 1e-6)
        x, m, tr = sv.gmres(1, b, tol=tol, restart=p.n_var)
    first = int(np.argmax(trace < tol)) + 1
    assert m == first
    np.testing.assert_array_equal(tr, trace[:m])
    r = np.linalg.norm(b - op.matvec(1, x))
    assert abs(r - tr[-1]) <= 1e-6 * tr[-1]


@pytest.mark.parametrize('steps', [1, 26, 40])
def test_residual_above_the_fused_gram_schmidt(ctx, steps):
    """4,693 unknowns: modified Gram-Schmidt vector by vector, norm partials over many blocks.
    The same identity; the explicit residual is formed with the oracle's operator."""
    p0 = configs.na_sphere(radius=35.0, n_freq=2, method='iterative')
    text = p0.to_keyword_text()
    p, s = Problem.from_keyword_text(text), model.System.from_keywords(keywords.read_keyword_text(text))
    rng = np.random.default_rng(steps)
    b = rng.standard_normal(p.n_var) + 1j * rng.standard_normal(p.n_var)
    with Solver(p, ctx=ctx, store_t=True) as sv:
        _, n, trace = sv.gmres(1, b, tol=3e-2 * np.linalg.norm(b), restart=500)
        assert n >= 40
        tol = trace[steps - 1] * (1.0 + 1e-6)
        x, m, tr = sv.gmres(1, b, tol=tol, restart=500)
    assert m == int(np.argmax(trace < tol)) + 1
    r = np.linalg.norm(b - model.Operator(s).matvec(1, x))
    assert abs(r - tr[-1]) <= 1e-6 * tr[-1]
