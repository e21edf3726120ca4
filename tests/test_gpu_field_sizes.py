"""Field and density at the numbers of points and atoms where the kernel changes
path: one point, block edges, atoms split over blocks with a remainder, one and two
points a thread; near, damped, undamped and vanishing pairs, points on atoms.

Against the oracle, norm-wise to 1e-12 as in the analysis tests; the density element
by element to 1e-10 of the sum of its terms' magnitudes (an exponential's relative error
is u^2 eps, at most 745 eps = 2e-13).
"""
import numpy as np
import pytest

from oracle.analysis import field_and_density
from plasmonx_b200 import configs
from plasmonx_b200.solver import Context, Solver

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def ctx():
    c = Context(0)
    yield c
    c.close()


@pytest.mark.parametrize('metal,radius,n_points', [
    ('Na', 8.0, 1), ('Ag', 6.0, 127), ('Ag', 8.0, 128), ('Ag', 8.0, 129), ('Na', 12.0, 257), ('Ag', 12.0, 3375),
    ('Au', 12.0, 40001), ('Ag', 6.0, 151552), ('Na', 8.0, 151809)])
def test_points_and_atoms(ctx, metal, radius, n_points):
    p = configs.particle(metal, 'sphere', radius, n_freq=1, method='iterative')
    rng = np.random.default_rng(n_points)
    x = rng.standard_normal(p.n_var) + 1j * rng.standard_normal(p.n_var)
    ext = np.abs(p.coord).max()
    pts = rng.uniform(-1.2 * ext, 1.2 * ext, size=(n_points, 3))
    pts[::7] *= 12.0                                       # undamped and vanishing pairs
    k = min(5, n_points)
    pts[:k] = p.coord[:k]                                  # on atoms
    rq, rmu = p.r_q[p.atom_types], p.r_mu[p.atom_types]
    fmu = p.model == 'wfqfmu'
    with Solver(p, ctx=ctx, store_t=False) as sv:
        f, d = sv.field_at_points(1, x, pts)
    fr = np.concatenate([field_and_density(p.coord, rq, rmu, x, p.e0, 1, c, fmu)[0]
                         for c in np.array_split(pts, max(1, n_points // 5000))])
    dr = np.concatenate([field_and_density(p.coord, rq, rmu, x, p.e0, 1, c, fmu)[1]
                         for c in np.array_split(pts, max(1, n_points // 5000))])
    xa = np.abs(x).max() * np.ones_like(x)
    scale = np.abs(field_and_density(p.coord, rq, rmu, xa, p.e0, 1, pts[:200], False)[1])
    assert np.linalg.norm(f - fr) <= 1e-12 * np.linalg.norm(fr)
    assert np.linalg.norm(d - dr) <= 1e-12 * np.linalg.norm(dr)
    if not fmu:
        assert np.all(np.abs(d - dr)[:200] <= 1e-10 * scale + 1e-300)
