"""Schedule of the tensor-core contraction: fewer tiles than SMs (runs of k-tiles
across tiles), one tile, tiles shorter than a run, a full wave plus a remainder,
two column tiles, one and two accumulator sets (128 columns a tile and above).

Element by element against the FP64 contraction, with the bound of the arithmetic:
one BF16 product rounds each operand to 2^-9 (2^-8 (1 + 2^-10) of |T| |x|), three
products keep each operand to 2^-18 and drop low x low (3 x 2^-18), and FP32 sums of
n terms add at most n 2^-24; sodium's T is positive, so |T| |x| is T |x|.
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


def _check(ctx, p, counts):
    with Solver(p, ctx=ctx, store_t=True) as sv:
        for count in counts:
            X = np.random.default_rng(count).standard_normal((count, p.n_var))
            ref, scale = sv.contract(X, 'fp64'), sv.contract(np.abs(X), 'fp64')
            for how, bar in (('bf16x3', 3 * 2.0 ** -18), ('bf16', 2.0 ** -8 * (1 + 2.0 ** -10))):
                err = np.abs(sv.contract(X, how) - ref) / scale
                assert err.max() <= bar + p.n_var * 2.0 ** -24, (count, how, err.max())


@pytest.mark.parametrize('radius', [8.0, 12.0, 14.0, 20.0, 28.0])
def test_fewer_tiles_than_sms(ctx, radius):
    _check(ctx, configs.na_sphere(radius=radius, n_freq=1), [1, 2, 15, 17, 32, 33, 64, 66, 128, 130, 256, 258, 402])


def test_full_wave_and_remainder(ctx):
    p = configs.na_sphere(radius=57.0, n_freq=1)
    assert 2 * ((p.n_var + 255) // 256) > 148
    _check(ctx, p, [4, 300])
