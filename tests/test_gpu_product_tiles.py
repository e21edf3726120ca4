"""FP64 products where their tiles change: chunks of 16 k and above (1,024 unknowns),
160,000 elements of a batch, batches of 8, 16 and 64 rows; matrix-free products of few and
of many blocks.  The tile decides nothing but the time: a column has the same bits whatever
batch it comes in, and its elements lie within n eps of |T| |x| of the exact sums.
"""
import numpy as np
import pytest

from oracle import keywords, model
from plasmonx_b200 import configs, geometry
from plasmonx_b200.solver import Context, Solver

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -52


@pytest.fixture(scope='module')
def ctx():
    c = Context(0)
    yield c
    c.close()


def _sodium(n):
    pts = geometry.sphere('bcc', 4.225, 25.0, 0.01, 1)
    pts = pts[np.argsort((pts ** 2).sum(1), kind='stable')][:n]
    return configs.build('wfq', pts, ['Na'], np.zeros(n, np.int32), configs.ev_grid(2.6, 2.7, 1))


@pytest.mark.parametrize('how,n', [('fp64', n) for n in (17, 255, 512, 893, 1023, 1024, 1025, 1088, 1089)] +
                         [('fp64_otf', n) for n in (17, 128, 129, 400, 893)])
def test_a_columns_bits_do_not_depend_on_the_tile(ctx, how, n):
    p = _sodium(n)
    T = model.t_full(model.System.from_keywords(keywords.read_keyword_text(p.to_keyword_text())))
    # the matrix-free product of up to eight real columns is another kernel
    counts = [9, 10, 15, 16, 17, 18, 33, 49, 64, 66, 130, 156, 180, 313] if how == 'fp64' else [9, 16, 18, 34, 50, 130, 300]
    X = np.random.default_rng(n).standard_normal((max(counts), n))
    with Solver(p, ctx=ctx, store_t=True) as sv:
        ref = sv.contract(X, how)
        for c in counts:
            np.testing.assert_array_equal(sv.contract(X[:c], how), ref[:c])
    assert np.all(np.abs(ref - X @ T) <= n * EPS * (np.abs(X) @ np.abs(T)))
