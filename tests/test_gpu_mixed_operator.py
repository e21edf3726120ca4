"""The mixed-precision operator A(w) = A0 + D(w) element by element: the folded tensor-core
operand (stored and generated T, one and two atom types, clusters of 32 atoms with a
remainder, a cluster without neighbours), the boundary-element operand, the diagonal that
the contraction's epilogue adds, its column tiles, and grouped launches.

No entry point returns the mixed product itself, but a solve of two inner steps does: with
v1 = b / ||b|| and the Jacobi preconditioner P its solution is
    x = P (a v1 + c w),   w = A P v1,
so a and c are fitted (two numbers) and the rest, x / P - a v1 - c w with the product w in
FP64, is c times the error of the mixed product.  The inner tolerance lies between the
residuals after one and two steps, which plain numpy gives.

Bound of an element of that error, from the arithmetic: operand and column keep 2^-18 each
and low x low (2^-18) is dropped -- one product keeps 2^-9 of each: 2^-8 (1 + 2^-10) --
FP32 sums of n terms add n 2^-24 and the FP32 basis 2^-23, all of |A0| |P v1|; two basis
vectors rounded to FP32 add 2^-23 (|a v1| + |c w|) and the fit spreads at most the norm of
that over v1 and w.  Rounding alone reaches 0.02-0.3 of the bound; a row, column block or
tile that is wrong exceeds it some thousandfold, a single element where it counts more than
the other elements' rounding.
"""
import numpy as np
import pytest

from oracle import keywords, model
from plasmonx_b200 import bem, configs, geometry
from plasmonx_b200.inputs import Problem
from plasmonx_b200.solver import Batch, Context, Solver

pytestmark = pytest.mark.gpu

OPERAND = {'mixed_bf16x3': 3 * 2.0 ** -18, 'mixed_bf16': 2.0 ** -8 * (1 + 2.0 ** -10)}


@pytest.fixture(scope='module')
def ctx():
    c = Context(0)
    yield c
    c.close()


def problem(kind, n, n_freq, shuffle=False):
    """n atoms nearest the origin of a lattice, an alloy bow-tie of edge n, or sodium with its
    last atom out of every other's reach; n_freq neighbouring frequencies."""
    ev = {'ag': 3.4, 'na': 2.6, 'far': 2.6, 'bowtie': 2.9}[kind]
    freqs = configs.ev_grid(ev, ev * (1 + 1e-5 * n_freq), n_freq)
    rng = np.random.default_rng(n)
    if kind == 'bowtie':
        pts, types = geometry.bowtie(4.08, float(n), 10.0, 6.0, 0.01, 1)
        order = rng.permutation(len(pts)) if shuffle else np.arange(len(pts))
        p = configs.build('wfqfmu', pts[order], ['Ag', 'Au'], types[order], freqs)
    else:
        lat, a = ('fcc', 4.086) if kind == 'ag' else ('bcc', 4.225)
        pts = geometry.sphere(lat, a, 30.0, 0.01, 1)
        pts = pts[np.argsort((pts ** 2).sum(1), kind='stable')][:n]
        if kind == 'far':
            pts[-1] = [500.0, 3.0, -2.0]
        if shuffle:
            pts = pts[rng.permutation(n)]
        p = configs.build('wfqfmu' if kind == 'ag' else 'wfq', pts, ['Ag' if kind == 'ag' else 'Na'],
                          np.zeros(n, np.int32), freqs)
    text = p.to_keyword_text()
    return Problem.from_keyword_text(text), model.System.from_keywords(keywords.read_keyword_text(text))


class Dense:
    """A0 and D(w) of an atomistic system: plain numpy on the oracle's matrices."""

    def __init__(self, s):
        self.s, self.n, N = s, s.n_var, s.n_q
        op = model.Operator(s)
        self.T, self.K = op.T, op.K
        C = self.K if not s.heterogeneous else 0.5 * (self.K + self.K.T)
        self.A0 = self.T.copy()
        self.A0[:N] = C @ self.T[:N] - C.sum(1)[:, None] * self.T[:N]
        self.b = [op.rhs(f) for f in range(len(s.freqs))]

    def cross(self, f):
        """1/2 (w_j / w_i - 1) K_ji of atoms of different types."""
        w = model.drude_w(self.s, self.s.freqs[f])[self.s.types]
        return 0.5 * (w[None, :] / w[:, None] - 1.0) * self.K.T

    def apply(self, f, x):
        y = self.A0 @ x
        if self.s.heterogeneous:
            s, X = self.T[:self.s.n_q] @ x, self.cross(f)
            y[:self.s.n_q] += X @ s - X.sum(1) * s
        return y + self.shift(f) * x

    def shift(self, f):
        return model.diagonal(self.s, f)

    def inverse_diagonal(self, f):
        d = np.diag(self.A0) + self.shift(f)
        if self.s.heterogeneous:
            N, X = self.s.n_q, self.cross(f)
            d[:N] += np.einsum('ij,ji->i', X, self.T[:N, :N]) - X.sum(1) * np.diag(self.T)[:N]
        return 1.0 / d

    def magnitude(self, f, x):
        """Sum of the magnitudes of the products behind every element (|x|: real + imaginary)."""
        x = np.abs(x.real) + np.abs(x.imag)
        y = np.abs(self.A0) @ x
        if self.s.heterogeneous:
            s, X = np.abs(self.T[:self.s.n_q]) @ x, np.abs(self.cross(f))
            y[:self.s.n_q] += X @ s + X.sum(1) * s
        return y


class DenseBem:
    """D + z(w) of a boundary-element surface, through the library's FP64 products."""

    def __init__(self, sv):
        self.n = sv.n_var
        self.A0 = sv.contract(np.eye(self.n), 'fp64').T
        e = np.zeros(self.n, complex)
        e[0] = 1.0
        self.z = [sv.matvec(f, e)[0] - self.A0[0, 0] for f in range(len(sv.freqs))]
        self.b = [sv.rhs(f) for f in range(len(sv.freqs))]

    def apply(self, f, x):
        return self.A0 @ x + self.z[f] * x

    def inverse_diagonal(self, f):
        return 1.0 / (np.diag(self.A0) + self.z[f])

    def magnitude(self, f, x):
        return np.abs(self.A0) @ (np.abs(x.real) + np.abs(x.imag))


class TwoSteps:
    """The first two inner steps of column (f, pol): basis, product, residuals / ||b||."""

    def __init__(self, d, f, pol):
        self.d, self.f = d, f
        b = d.b[f][:, pol]
        self.P = d.inverse_diagonal(f)
        self.v1 = b / np.linalg.norm(b)
        self.w = d.apply(f, self.P * self.v1)
        v2 = self.w - (self.v1.conj() @ self.w) * self.v1
        w2 = d.apply(f, self.P * (v2 / np.linalg.norm(v2)))
        lsq = lambda M: np.linalg.norm(self.v1 - M @ np.linalg.lstsq(M, self.v1, rcond=None)[0])   # noqa: E731
        self.r1 = lsq(self.w[:, None])
        self.r2 = lsq(np.stack([self.w, w2], 1))

    def bound(self, precision, a, c):
        d = self.d
        eta = OPERAND[precision] + d.n * 2.0 ** -24 + 2.0 ** -23
        e = np.abs(c) * eta * d.magnitude(self.f, self.P * self.v1)
        return e + 2.0 ** -23 * (np.abs(a * self.v1) + np.abs(c * self.w))

    def check(self, x, precision):
        u = x / self.P
        M = np.stack([self.v1, self.w], 1)
        a, c = np.linalg.lstsq(M, u, rcond=None)[0]
        bar = self.bound(precision, a, c)
        q = np.abs(np.linalg.qr(M)[0])
        err, bar = np.abs(u - M @ np.array([a, c])), bar + np.linalg.norm(bar) * q.sum(1)
        assert (err <= bar).all(), (int(np.argmax(err - bar)), (err / np.maximum(bar, 1e-300)).max())


def window(steps):
    """An inner tolerance that every column passes in its second step."""
    lo, hi = max(s.r2 for s in steps), min(s.r1 for s in steps)
    assert hi > 1.02 * lo, (lo, hi)
    return np.sqrt(lo * hi)


def solve_two(sv, steps, pol, precision, mode='iterative'):
    out = sv.solve(mode=mode, precision=precision, pol_mask=1 << pol, tol=1e-300, inner_krylov=2,
                   inner_tol=window(steps), max_outer=1, want_x=True)
    assert (out['steps'][:, pol] == 2).all(), out['steps'][:, pol]
    return out['x'][:, :, pol]


ATOMS = [('na', 31, 1, False), ('na', 450, 9, True), ('far', 33, 2, False), ('ag', 13, 1, False), ('ag', 33, 9, True),
         ('ag', 200, 65, False), ('ag', 321, 129, True), ('bowtie', 16, 2, False), ('bowtie', 22, 65, True)]


@pytest.mark.parametrize('precision', sorted(OPERAND))
@pytest.mark.parametrize('store_t', [True, False])
@pytest.mark.parametrize('kind,n,n_freq,shuffle', ATOMS)
def test_folded_operator(ctx, kind, n, n_freq, shuffle, store_t, precision):
    p, s = problem(kind, n, n_freq, shuffle)
    d = Dense(s)
    look = sorted({0, n_freq // 2, n_freq - 1})
    with Solver(p, ctx=ctx, store_t=store_t) as sv:
        for pol in range(3):
            steps = {f: TwoSteps(d, f, pol) for f in look}
            x = solve_two(sv, list(steps.values()), pol, precision, 'iterative' if store_t else 'iterative on the fly')
            for f in look:
                steps[f].check(x[f], precision)


@pytest.mark.parametrize('precision', sorted(OPERAND))
@pytest.mark.parametrize('shape,n,n_freq', [('sphere', 500, 1), ('rod', 720, 9), ('sphere', 980, 129)])
def test_boundary_element_operator(ctx, shape, n, n_freq, precision):
    p = bem.bem_surface(n, shape=shape, n_freq=301, polarization='all', method='iterative')
    with Solver(p, ctx=ctx) as sv:
        k = 150
        sv.set_frequencies(np.full(n_freq, p.freqs[k]) * (1 + 1e-6 * np.arange(n_freq)),
                           p.alpha_w[:, k:k + 1] * (1 + 1e-6 * np.arange(n_freq)))
        d = DenseBem(sv)
        look = sorted({0, n_freq // 2, n_freq - 1})
        for pol in range(3):
            steps = {f: TwoSteps(d, f, pol) for f in look}
            x = solve_two(sv, list(steps.values()), pol, precision)
            for f in look:
                steps[f].check(x[f], precision)


GROUP = [('ag', 200, 20), ('na', 31, 1), ('na', 1500, 3), ('ag', 33, 65), ('bowtie', 16, 9), ('na', 450, 129), ('ag', 13, 2)]


@pytest.mark.parametrize('members', [[0, 1], [1, 6], [2, 3, 4], [0, 1, 2, 3, 4, 5], [0, 1, 2, 3, 4, 5, 6]])
def test_grouped_launches(ctx, members):
    """Geometries of very different order and width in one launch (seven: in two).  A batch
    returns no solution but its polarisability, sum_i r_i q_i / E0 (+ dipoles): compared with
    the single solve's within twice the bound above, summed with the same weights."""
    solvers, batches, refs = [], [], []
    try:
        for m in members:
            kind, n, n_freq = GROUP[m]
            p, s = problem(kind, n, n_freq)
            d = Dense(s)
            sv = Solver(p, ctx=ctx, store_t=True)
            solvers.append(sv)
            steps = [TwoSteps(d, f, 0) for f in sorted({0, n_freq // 2, n_freq - 1})]
            x = solve_two(sv, steps, 0, 'mixed_bf16x3')
            refs.append((s, steps, x))
            b = Batch(sv, precision='mixed_bf16x3', inner_krylov=2, inner_tol=window(steps), max_outer=1)
            batches.append(b)
            b.add(m, p.freqs, p.alpha_w, pol_mask=1, tol=1e-300)
        Batch.step_group(batches)
        for m, b, (s, steps, x) in zip(members, batches, refs):
            out = b.take(m)
            assert (out['steps'][:, 0] == 2).all()
            for st in steps:
                f, N = st.f, s.n_atoms
                u = x[f] / st.P
                M = np.stack([st.v1, st.w], 1)
                a, c = np.linalg.lstsq(M, u, rcond=None)[0]
                bar = st.bound('mixed_bf16x3', a, c)
                # the two solves' coefficients differ as the least-squares problem does
                bar = np.abs(st.P) * (bar + np.linalg.norm(bar) * np.abs(np.linalg.qr(M)[0]).sum(1) *
                                      (1 + np.linalg.cond(M)))
                ref = model.polar(s, np.stack([x[f]] * 3, 1))[:, 0]
                got = out['polar'][f][:, 0]
                for k in range(3):
                    tol = (np.abs(s.coord[:, k]) * bar[:N]).sum() / s.e0
                    if s.model == 'wfqfmu':
                        tol += bar[N + k::3][:N].sum() / s.e0
                    assert abs(got[k] - ref[k]) <= 2.0 * tol, (m, f, k, abs(got[k] - ref[k]), tol)
    finally:
        for b in batches:
            b.close()
        for sv in solvers:
            sv.close()


def test_generated_rows_in_several_batches(ctx):
    """Sodium spheres of more atoms than the matrix-free fold generates rows for at a time
    (750 million elements): the second batch's rows against those folded from a stored T.
    Both operands round the same sums (to 1e-12) to 16 bits, so an element of x may differ by
    the operand's rounding at most: 2^-15 of the largest."""
    p = configs.na_sphere(radius=64.0, n_freq=1)
    assert p.n_var ** 2 > 750e6
    kw = dict(precision='mixed_bf16x3', pol_mask=1, tol=1e-300, inner_krylov=4, inner_tol=1e-12, max_outer=1, want_x=True)
    x = []
    for store_t, mode in ((True, 'iterative'), (False, 'iterative on the fly')):
        with Solver(p, ctx=ctx, store_t=store_t) as sv:
            x.append(sv.solve(mode=mode, **kw)['x'][0, :, 0])
    assert np.abs(x[0]).max() > 0
    assert np.abs(x[1] - x[0]).max() <= 2.0 ** -15 * np.abs(x[0]).max()
