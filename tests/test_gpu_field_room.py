"""Field and density on small grids where there is little or no room for the sums of the
atoms' parts: the call takes what its inputs and outputs take, and the values are those of
a context with room, to the rounding of sums over N atoms of terms that partly cancel
(held to the 1e-12 of the analysis tests).
"""
import numpy as np
import pytest

from plasmonx_b200 import configs
from plasmonx_b200.solver import Context, Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('metal,radius,n_points', [('Na', 12.0, 1), ('Ag', 12.0, 500), ('Ag', 16.0, 3375)])
@pytest.mark.parametrize('spare', [0, 0.3, 0.6])
def test_little_room_for_partial_sums(metal, radius, n_points, spare):
    p = configs.particle(metal, 'sphere', radius, n_freq=1, method='iterative')
    rng = np.random.default_rng(n_points)
    x = rng.standard_normal(p.n_var) + 1j * rng.standard_normal(p.n_var)
    pts = rng.uniform(-1.2, 1.2, size=(n_points, 3)) * np.abs(p.coord).max()
    c = Context(0)
    with Solver(p, ctx=c, store_t=False) as sv:
        held = c.bytes_in_use
        f0, d0 = sv.field_at_points(2, x, pts)
    c.close()
    parts = -(-p.n_atoms // 128)                       # at most: a tile of 128 atoms each
    assert parts > 1
    room = 16 * p.n_var + 8 * (3 + 6 + 2) * n_points + int(spare * 64 * n_points * parts)
    c = Context(0, hbm_budget=held + room)
    try:
        with Solver(p, ctx=c, store_t=False) as sv:
            f, d = sv.field_at_points(2, x, pts)
    finally:
        c.close()
    assert np.linalg.norm(f - f0) <= 1e-12 * np.linalg.norm(f0)
    assert np.linalg.norm(d - d0) <= 1e-12 * np.linalg.norm(d0)
