"""Plain GMRES where its steps change kernel: modified Gram-Schmidt in one launch with one,
two and four groups of 1,024 rows a column (1,025 to 4,096 unknowns) and above it, and a
matrix-free solve whose batch falls from the tiled product (more than four columns) to the
one with a warp per atom as columns converge.

As in the Arnoldi tests, the explicit residual ||b - A x|| with the oracle's operator equals
the recurrence's last residual up to rounding of the order of 1e-15 ||A|| ||x|| against a
residual of at least 1e-6 ||b||: held to 1e-6 of it, for the matrix-free columns to 1e-4.
"""
import functools

import numpy as np
import pytest

from oracle import keywords, model
from plasmonx_b200 import configs, geometry
from plasmonx_b200.inputs import Problem
from plasmonx_b200.solver import Context, Solver

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def ctx():
    c = Context(0)
    yield c
    c.close()


def _both(p):
    text = p.to_keyword_text()
    return Problem.from_keyword_text(text), model.System.from_keywords(keywords.read_keyword_text(text))


@functools.lru_cache(maxsize=1)
def _sodium(n):
    pts = geometry.sphere('bcc', 4.225, 36.0, 0.01, 1)
    pts = pts[np.argsort((pts ** 2).sum(1), kind='stable')][:n]
    p, s = _both(configs.build('wfq', pts, ['Na'], np.zeros(n, np.int32), configs.ev_grid(2.6, 2.7, 2)))
    return p, model.Operator(s)


@pytest.mark.parametrize('n', [1023, 1024, 1025, 2047, 2048, 2049, 3073, 4095, 4096, 4097])
def test_steps_by_order(ctx, n):
    p, op = _sodium(n)
    assert p.n_var == n
    rng = np.random.default_rng(n)
    b = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    with Solver(p, ctx=ctx, store_t=True) as sv:
        _, most, trace = sv.gmres(1, b, tol=3e-2 * np.linalg.norm(b), restart=500)
        assert most >= 26
        for steps in (1, 2, 3, 24, 25, 26):
            tol = trace[steps - 1] * (1.0 + 1e-6)
            x, m, tr = sv.gmres(1, b, tol=tol, restart=500)
            assert m == int(np.argmax(trace < tol)) + 1
            np.testing.assert_array_equal(tr, trace[:m])
            r = np.linalg.norm(b - op.matvec(1, x))
            assert abs(r - tr[-1]) <= 1e-6 * tr[-1]


@pytest.mark.parametrize('metal,n_freq', [('Na', 2), ('Na', 7), ('Ag', 3)])
def test_matrix_free_batch_that_shrinks(ctx, metal, n_freq):
    p, s = _both(configs.particle(metal, 'rod', 7.0, n_freq=n_freq, method='iterative on the fly'))
    op = model.Operator(s)
    tol = 1e-6 * np.linalg.norm(op.rhs(0)[:, 0])
    with Solver(p, ctx=ctx, store_t=False) as sv:
        out = sv.solve(tol=tol, max_krylov=p.n_var, pol_mask=7, want_x=True)
    assert (out['status'] == 0).all()
    finish = np.sort(out['steps'].ravel())
    assert finish[-4] > finish[0]                        # the batch is down to four before the end
    for f in range(n_freq):
        b = op.rhs(f)
        for pol in range(3):
            r = np.linalg.norm(b[:, pol] - op.matvec(f, out['x'][f, :, pol]))
            assert r <= tol * (1.0 + 1e-4)
