"""The folded tensor-core operand, stored and generated T, one and two atom types,
numbers of atoms around the clusters of 32, atoms in no spatial order.

An inner solve to 1e-3 on an operator that is off by ~1e-5 (BF16x3) takes the steps the
FP64 operator takes, give or take one where the last residual lands next to the
tolerance; a wrong element of the operand would not.
"""
import numpy as np
import pytest

from plasmonx_b200 import configs, geometry
from plasmonx_b200.solver import Context, Solver

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def ctx():
    c = Context(0)
    yield c
    c.close()


def _cluster(kind, n, shuffle):
    """The n lattice sites nearest the origin (Ag wFQFMu, Na wFQ), or an alloy bow-tie."""
    rng = np.random.default_rng(n)
    if kind == 'bowtie':
        pts, types = geometry.bowtie(4.08, 24.0, 10.0, 6.0, 0.01, 1)
        order = rng.permutation(len(pts)) if shuffle else np.arange(len(pts))
        return configs.build('wfqfmu', pts[order], ['Ag', 'Au'], types[order], configs.ev_grid(2.0, 4.5, 3))
    lat, a = ('fcc', 4.086) if kind == 'ag' else ('bcc', 4.225)
    pts = geometry.sphere(lat, a, 30.0, 0.01, 1)
    pts = pts[np.argsort((pts ** 2).sum(1), kind='stable')][:n]
    if shuffle:
        pts = pts[rng.permutation(n)]
    if kind == 'ag':
        return configs.build('wfqfmu', pts, ['Ag'], np.zeros(n, np.int32), configs.ev_grid(3.0, 4.5, 3))
    return configs.build('wfq', pts, ['Na'], np.zeros(n, np.int32), configs.ev_grid(2.0, 4.0, 3))


@pytest.mark.parametrize('kind,n,shuffle', [('ag', 13, False), ('ag', 32, False), ('ag', 33, True), ('ag', 200, False),
                                            ('ag', 321, True), ('na', 31, False), ('na', 450, True),
                                            ('bowtie', 0, False), ('bowtie', 0, True)])
@pytest.mark.parametrize('store_t', [True, False])
def test_inner_steps_match_the_fp64_operator(ctx, kind, n, shuffle, store_t):
    p = _cluster(kind, n, shuffle)
    mode = 'iterative' if store_t else 'iterative on the fly'
    with Solver(p, ctx=ctx, store_t=store_t) as sv:
        tol = 2e-3 * np.linalg.norm(sv.rhs(0, 1)[:, 0])
        kw = dict(mode=mode, pol_mask=1, tol=tol, inner_krylov=p.n_var, inner_tol=1e-3, max_outer=1)
        ref = sv.solve(precision='fp64_refined', **kw)
        got = sv.solve(precision='mixed_bf16x3', **kw)
    assert np.all(np.abs(got['steps'] - ref['steps']) <= 1), (got['steps'][:, 0], ref['steps'][:, 0])


def test_little_room_folds_in_smaller_batches(ctx):
    """1,961 atoms: the clusters' coefficients take about 13 MB together and 0.2 MB one by one.
    The batch a cluster is folded in does not change its sums: the solution keeps its bits."""
    p = configs.ag_sphere(radius=20.0, n_freq=1, method='iterative')
    kw = dict(precision='mixed_bf16x3', pol_mask=1, want_x=True, max_outer=2, inner_krylov=16)
    probe = Context(0)
    with Solver(p, ctx=probe, store_t=True) as sv:
        ref = sv.solve(**kw)
        held = probe.bytes_in_use
    probe.close()
    tight = Context(0, hbm_budget=held + 5_000_000)
    with Solver(p, ctx=tight, store_t=True) as sv:
        got = sv.solve(**kw)
    tight.close()
    np.testing.assert_array_equal(got['status'], ref['status'])
    np.testing.assert_array_equal(got['x'], ref['x'])
