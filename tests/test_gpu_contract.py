"""Stored-T FP64 products at the edges of their row tiles (2 to 16, 32, 48, 64 and
beyond) and the conductance rows at warp edges.

The products' values: T itself from unit columns, X T in numpy; sums of n <= 893 terms
carry n eps at most (2e-13).  A column does not depend on its batch, bit for bit, over
all the kernels.  The conductance: the stored pairs are those whose Fermi factor is not
zero in double precision, counted by numpy over all pairs.
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


@pytest.mark.parametrize('radius', [8.0, 12.0, 20.0])
def test_products_and_their_batches(ctx, radius):
    p = configs.na_sphere(radius=radius, n_freq=1)
    n = p.n_var
    X = np.random.default_rng(n).standard_normal((130, n))
    with Solver(p, ctx=ctx, store_t=True) as sv:
        T = sv.contract(np.eye(n), 'fp64')
        full = sv.contract(X, 'fp64')
        ref = X @ T
        assert np.max(np.linalg.norm(full - ref, axis=1) / np.linalg.norm(ref, axis=1)) < 2e-13
        for count in (1, 2, 3, 4, 6, 7, 8, 10, 12, 14, 16, 17, 18, 32, 33, 34, 48, 49, 50, 64, 65, 66, 128):
            np.testing.assert_array_equal(sv.contract(X[:count], 'fp64'), full[:count], err_msg=str(count))


@pytest.mark.parametrize('problem', [
    lambda: configs.na_sphere(radius=3.0, n_freq=1), lambda: configs.na_sphere(radius=8.0, n_freq=1),
    lambda: configs.na_sphere(radius=20.0, n_freq=1), lambda: configs.ag_sphere(radius=14.0, n_freq=1, jitter=0.01),
    lambda: configs.agau_bowtie(edge=28.0, n_freq=1, jitter=0.01)])
def test_conductance_pairs(ctx, problem):
    p = problem()
    t = p.atom_types
    d = p.coord[:, None, :] - p.coord[None, :, :]
    r = np.sqrt((d * d).sum(-1))
    np.fill_diagonal(r, 1.0)
    u = p.fermi_d[t[:, None], t] * (r / (p.fermi_s[t[:, None], t] * p.r0[t[:, None], t]) - 1.0)
    k = 1.0 - 1.0 / (1.0 + np.exp(-u)) != 0.0
    np.fill_diagonal(k, False)
    with Solver(p, ctx=ctx, store_t=False) as sv:
        assert sv.k_nnz == np.count_nonzero(k | k.T)
