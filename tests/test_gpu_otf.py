"""Matrix-free FP64 products at the sizes where their kernels change path: one
to four columns (warps per target atom 8, 4, 2, 1 with the number of atoms),
the tiled form's row tiles (16, 32, 48, 64 and two of them), ragged numbers of
atoms, near and undamped distant pairs, one and two atom types.

Against the product with the stored T, which evaluates every pair by the
unshortened formulas.  Elements agree to a few ulp and a sum of n terms carries
a rounding of about sqrt(n) eps (1.4e-14 at 15,000 unknowns): held to 1e-13.
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


PROBLEMS = {
    'ag_135': lambda: configs.ag_sphere(radius=8.0, n_freq=1, jitter=0.01),
    'ag_959': lambda: configs.ag_sphere(radius=16.0, n_freq=1, jitter=0.01),
    'ag_1961': lambda: configs.ag_sphere(radius=20.0, n_freq=1, jitter=0.01),
    'ag_3805': lambda: configs.ag_sphere(radius=25.0, n_freq=1, jitter=0.01),
    'bowtie_700': lambda: configs.agau_bowtie(edge=28.0, n_freq=1, jitter=0.01),
    'na_59': lambda: configs.na_sphere(radius=8.0, n_freq=1),
    'na_2421': lambda: configs.na_sphere(radius=28.0, n_freq=1),
}


@pytest.mark.parametrize('count', [1, 2, 3, 5, 8, 9, 16, 17, 32, 33, 48, 49, 65])
@pytest.mark.parametrize('name', sorted(PROBLEMS))
def test_generated_tiles_match_the_stored_matrix(ctx, name, count):
    if name == 'ag_3805' and count not in (1, 8, 33):
        pytest.skip('one size per kernel for the largest geometry')
    p = PROBLEMS[name]()
    X = np.random.default_rng(count).standard_normal((count, p.n_var))
    with Solver(p, ctx=ctx, store_t=True) as sv:
        ref = sv.contract(X, 'fp64')
        got = sv.contract(X, 'fp64_otf')
    err = np.linalg.norm(got - ref, axis=1) / np.linalg.norm(ref, axis=1)
    assert err.max() < 1e-13, err.max()


@pytest.mark.parametrize('few,many', [(2, 8), (4, 6), (10, 34), (16, 64), (30, 130)])
def test_a_column_does_not_depend_on_its_batch(ctx, few, many):
    """Within the few-column kernel and within the tiled one, bit for bit."""
    p = PROBLEMS['bowtie_700']()
    X = np.random.default_rng(1).standard_normal((many, p.n_var))
    with Solver(p, ctx=ctx, store_t=False) as sv:
        np.testing.assert_array_equal(sv.contract(X[:few], 'fp64_otf'), sv.contract(X, 'fp64_otf')[:few])


@pytest.mark.parametrize('count', [9, 16, 31, 32])
def test_a_few_columns_need_no_scratch(ctx, count):
    """Up to 16 complex columns go on, four at a time, where the budget has no room for the
    tiled form's partial sums (4.7 MB at 16 columns here); the operands take 0.28 MB."""
    p = PROBLEMS['ag_135']()
    X = np.random.default_rng(count).standard_normal((count, p.n_var))
    with Solver(p, ctx=ctx, store_t=False) as sv:
        ref = sv.contract(X, 'fp64_otf')
    probe = Context(0)
    with Solver(p, ctx=probe, store_t=False):
        held = probe.bytes_in_use
    probe.close()
    tight = Context(0, hbm_budget=held + 600_000)
    with Solver(p, ctx=tight, store_t=False) as sv:
        got = sv.contract(X, 'fp64_otf')
    tight.close()
    err = np.linalg.norm(got - ref, axis=1) / np.linalg.norm(ref, axis=1)
    assert err.max() < 1e-13, err.max()
