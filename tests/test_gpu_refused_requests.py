"""Requests that the budget refuses: a frequency grid leaves the geometry without
frequencies (and says so), a request of a batch leaves the batch as it was -- its tables,
slots and results are those of a batch that never saw the request.
"""
import numpy as np
import pytest

from plasmonx_b200 import _lib, bem, configs
from plasmonx_b200.solver import Batch, Context, Solver

pytestmark = pytest.mark.gpu

KINDS = {
    'na': lambda f: configs.na_sphere(radius=9.0, n_freq=f),
    'bowtie': lambda f: configs.agau_bowtie(edge=18.0, n_freq=f),
    'dpcm': lambda f: bem.bem_surface(500, n_freq=f, polarization='x', method='iterative'),
}


@pytest.mark.parametrize('kind', sorted(KINDS))
def test_a_refused_grid_leaves_no_frequencies(kind):
    p = KINDS[kind](3)
    wide = np.tile(p.freqs, 150000)                    # tables of 7 to 58 MB
    alpha = None if p.alpha_w is None else np.tile(p.alpha_w, (1, 150000))
    c = Context(0)
    with Solver(p, ctx=c, store_t=None if kind == 'dpcm' else True) as sv:
        held = c.bytes_in_use
    c.close()
    c = Context(0, hbm_budget=held + 4000000)
    try:
        with Solver(p, ctx=c, store_t=None if kind == 'dpcm' else True) as sv:
            x = np.random.default_rng(0).standard_normal(sv.n_var) + 0j
            y = sv.matvec(1, x)
            with pytest.raises(_lib.PlxError) as e:
                sv.set_frequencies(wide, alpha)
            assert e.value.code == 4
            with pytest.raises(_lib.PlxError) as e:
                sv.matvec(1, x)
            assert e.value.code == 1
            sv.set_frequencies(p.freqs, p.alpha_w)
            np.testing.assert_array_equal(sv.matvec(1, x), y)
    finally:
        c.close()


@pytest.mark.parametrize('kind', sorted(KINDS))
@pytest.mark.parametrize('when', ['first', 'later'])
def test_a_refused_request_leaves_the_batch_as_it_was(kind, when):
    p, more = KINDS[kind](5), KINDS[kind](400)
    kw = dict(pol_mask=1, tol=1e-9)
    store = None if kind == 'dpcm' else True

    def run(budget, refused):
        c = Context(0, hbm_budget=budget)
        peak = 0
        with Solver(p, ctx=c, store_t=store) as sv, Batch(sv, precision='mixed_bf16x3') as b:
            def attempt():
                with pytest.raises(_lib.PlxError) as e:
                    b.add(9, more.freqs, more.alpha_w, **kw)
                assert e.value.code == 4
            if refused and when == 'first':
                attempt()
            b.add(1, p.freqs, p.alpha_w, **kw)
            k = 0
            while b.active:
                b.step()
                k += 1
                if refused and when == 'later' and k == 1:
                    attempt()
                peak = max(peak, c.bytes_in_use)
            out = b.take(1)
            used = c.bytes_in_use
        c.close()
        return out, peak, used

    ref, _, _ = run(0, False)
    # the smallest budget (to a few per cent) that the five columns alone run in; the step's own
    # arrays are freed between calls, so it is found by trying
    lo, hi = 1 << 20, 1 << 28
    while hi > 1.05 * lo:
        mid = int((lo * hi) ** 0.5)
        try:
            run(mid, False)
            hi = mid
        except _lib.PlxError:
            lo = mid
    out, _, _ = run(hi, True)
    assert (out['status'] == 0).all()
    np.testing.assert_array_equal(out['results'], ref['results'])
    np.testing.assert_array_equal(out['steps'], ref['steps'])
