"""A call that the budget refuses half-way leaves the geometry as it was: once there is
room again (here a second geometry of the context is closed), the same call gives the
bits of a context that always had room.

The budgets run from the geometry alone to all that the call needs, so that every one of
its allocations is the refused one for some of them, the second half of a pair (operand
high and low, the two boundary-element products, the two diagonal parts) among them.
"""
import numpy as np
import pytest

from plasmonx_b200 import bem, configs
from plasmonx_b200.solver import Context, Solver

pytestmark = pytest.mark.gpu

MIXED = dict(precision='mixed_bf16x3', pol_mask=1, want_x=True, max_outer=2, inner_krylov=8)
CASES = {
    'ag': (lambda: configs.ag_sphere(radius=8.0, n_freq=1, method='iterative'), MIXED),
    'ag_generated': (lambda: configs.ag_sphere(radius=8.0, n_freq=1, method='iterative on the fly'), MIXED),
    'bowtie': (lambda: configs.agau_bowtie(edge=20.0, n_freq=1, method='iterative on the fly'), MIXED),
    'dpcm': (lambda: bem.bem_surface(500, n_freq=1, polarization='x', method='iterative'), MIXED),
    'ief_direct': (lambda: bem.bem_surface(300, variant='iefpcm', green='accurate', n_freq=1, polarization='x',
                                           method='inversion'), dict(pol_mask=1, want_x=True)),
}


def _refused(out):
    """The call met the budget (a solve that ran out of steps ran)."""
    return 'error' in out and out['error'].code in (3, 4)


def _need(p, kw):
    """Bytes of the geometry, and the room above it that the call takes (to a part in 32)."""
    c = Context(0)
    with Solver(p, ctx=c):
        held = c.bytes_in_use
    c.close()

    def runs(room):
        c = Context(0, hbm_budget=held + room)
        with Solver(p, ctx=c) as sv:
            out = sv.solve(**kw)
        c.close()
        return not _refused(out)

    lo, hi = 0, 1 << 20
    while not runs(hi):
        assert hi < 1 << 30
        lo, hi = hi, 2 * hi
    while hi - lo > hi // 32:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if runs(mid) else (mid, hi)
    return held, hi


@pytest.mark.parametrize('kind', sorted(CASES))
def test_a_refused_call_can_be_repeated(kind):
    make, kw = CASES[kind]
    p = make()
    held, need = _need(p, kw)
    c = Context(0)
    with Solver(p, ctx=c) as sv:
        ref = sv.solve(**kw)
    c.close()
    ballast = configs.na_sphere(radius=30.0, n_freq=1)               # T of 70 MB
    c = Context(0)
    with Solver(ballast, ctx=c, store_t=True):
        weight = c.bytes_in_use
    c.close()
    assert weight > need
    refused = 0
    for room in np.linspace(0, need, 33).astype(int):
        c = Context(0, hbm_budget=held + weight + int(room))
        try:
            with Solver(p, ctx=c) as sv:
                with Solver(ballast, ctx=c, store_t=True):
                    first = sv.solve(**kw)
                    if _refused(first):
                        refused += 1
                out = sv.solve(**kw)
                assert not _refused(out), (kind, room, out['error'])
                np.testing.assert_array_equal(out['status'], ref['status'])
                np.testing.assert_array_equal(out['x'], ref['x'])
        finally:
            c.close()
    assert refused >= 16
