"""The direct solve of the scalar-shift models where device memory is short: it takes the
Hessenberg reduction as long as three n x n matrices fit beside T (H, Q^T and one
frequency's triangular factor), the frequencies in as many waves as that needs, and gives
the bits it gives with all the room there is.  With less room the LU of every frequency
solves the same systems and leaves nothing of a reduction behind.
"""
import numpy as np
import pytest

from plasmonx_b200 import bem, configs
from plasmonx_b200.solver import Context, Solver

pytestmark = pytest.mark.gpu

CASES = {
    'na': lambda: configs.na_sphere(radius=16.0, n_freq=25, method='inversion', polarization='all'),
    'dpcm': lambda: bem.bem_surface(720, n_freq=40, method='inversion', polarization='all'),
}


def _solve(p, budget=0):
    c = Context(0, hbm_budget=budget)
    try:
        with Solver(p, ctx=c) as sv:
            held = c.bytes_in_use
            outs = [sv.solve(want_x=True) for _ in range(2)]
            return outs, held, c.bytes_in_use, sv.n_var
    finally:
        c.close()


@pytest.mark.parametrize('kind', sorted(CASES))
def test_three_matrices_beside_t_are_enough(kind):
    p = CASES[kind]()
    (ref, _), held, kept, n = _solve(p)
    cols = 3 * len(p.freqs)
    # the columns (right-hand sides, solutions, their potentials twice) and small tables
    columns = 4 * cols * 2 * n * 8 + (1 << 17)
    assert kept - held <= 2 * 8 * n * n + (1 << 16)              # what a solve leaves: H and Q^T
    outs, _, _, _ = _solve(p, held + columns + 3 * 8 * n * n + 8 * n)
    for out in outs:
        assert (out['status'] == 0).all()
        np.testing.assert_array_equal(out['x'], ref['x'])


@pytest.mark.parametrize('kind', sorted(CASES))
def test_less_room_leaves_no_reduction_behind(kind):
    p = CASES[kind]()
    (ref, _), held, _, n = _solve(p)
    cols = 3 * len(p.freqs)
    outs, held2, kept, _ = _solve(p, held + 2 * cols * 2 * n * 8 + int(2.8 * 8 * n * n))
    assert held2 == held and kept == held
    for out in outs:
        assert (out['status'] == 0).all()
        assert np.abs(out['x'] - ref['x']).max() <= 1e-9 * np.abs(ref['x']).max()
