"""Performance cases of the response solve, through the package's public entry points.

A case is a dict of plain values.  ``listed()`` gives the fixed ones, ``draw(rng)``
one more of the same ranges, ``prepare(case, seed)`` what a program holds before the
call (geometry, frequency grid, and for a resident geometry its ``Solver``), and
``run(state)`` one pass.  ``work(case)`` counts what a pass cannot do without and
``exact(case, seed)`` gives its outputs from plain torch in 64 bits.

Kinds:
  matvec    one product A(w) x, the call a host GMRES makes (stored T, or T generated)
  contract  S = T X of a few real columns with the stored FP64 T
  solve     a spectrum: resident geometry, or with ``fresh`` the geometry built,
            solved and released in the pass, as a program run once per geometry does
  bem       a spectrum of a boundary-element surface
  serve     continuous batching: one request per resident geometry, stepped together
  field     induced field and density of a solution on a cubic grid

Every iterative solve asks for a residual of ``rtol`` times the norm of its
right-hand side, so that two solves of one system agree far below the 1e-6 the
benchmark quotes.
"""
import math

import numpy as np
import torch

from plasmonx_b200 import analysis, bem, configs
from plasmonx_b200.solver import Batch, Context, Solver

JITTER = 0.01              # Angstrom, uniform, from the seed
LIGHT = 137.035227
TO_BOHR = 1.8897261254578281


def listed():
    return [
        # the smallest call: one product for a host-side GMRES on an 893-atom sodium sphere
        dict(name='matvec_na_893', kind='matvec', shape='na', size=20.0, otf=False),
        # the same product without a stored matrix: 1,961 silver atoms, tiles generated
        dict(name='matvec_otf_ag_1961', kind='matvec', shape='ag', size=20.0, otf=True),
        # three polarisations' columns against the stored FP64 T of 15,220 unknowns
        dict(name='contract_ag_3805', kind='contract', shape='ag', size=25.0, count=6),
        # the reference's own GMRES on memory: a sodium sphere's spectrum
        dict(name='gmres_na_893', kind='solve', shape='na', size=20.0, n_freq=61, pol='x', mode='iterative',
             precision='fp64', inner=0, inner_tol=0.0, rtol=1e-11, fresh=False),
        # a program run once: geometry, direct inversion of the whole grid, all polarisations
        dict(name='direct_na_893', kind='solve', shape='na', size=20.0, n_freq=61, pol='all', mode='inversion',
             precision='fp64', inner=0, inner_tol=0.0, rtol=0.0, fresh=True),
        # an ordinary spectrum on a resident silver sphere, mixed precision
        dict(name='mixed_ag_1961', kind='solve', shape='ag', size=20.0, n_freq=61, pol='x', mode='iterative',
             precision='mixed_bf16x3', inner=64, inner_tol=1e-4, rtol=2e-11, fresh=False),
        # the benchmark's silver sphere (41,892 unknowns) built and solved once, a block of its grid
        dict(name='fresh_ag_10473', kind='solve', shape='ag', size=35.0, n_freq=21, pol='x', mode='iterative',
             precision='mixed_bf16', inner=64, inner_tol=3e-2, rtol=2e-11, fresh=True),
        # the reference's on-the-fly GMRES on a small alloy bow-tie
        dict(name='otf_bowtie_700', kind='solve', shape='bowtie', size=28.0, n_freq=4, pol='x',
             mode='iterative on the fly', precision='fp64', inner=0, inner_tol=0.0, rtol=1e-11, fresh=False),
        # the matrix-free alloy bow-tie in mixed precision, resident operand
        dict(name='mixed_bowtie_3382', kind='solve', shape='bowtie', size=60.0, n_freq=21, pol='x',
             mode='iterative on the fly', precision='mixed_bf16x3', inner=256, inner_tol=1e-3, rtol=2e-11,
             fresh=False),
        # a boundary-element sphere of 8,000 tesserae over its whole window
        dict(name='bem_sphere_8000', kind='bem', shape='sphere', n_tess=8000, n_freq=301, pol='x',
             precision='mixed_bf16x3', rtol=1e-11),
        # the serving loop: requests on several resident geometries advanced together
        dict(name='serve_6', kind='serve', size=14.0, requests=6, n_freq=40, rtol=2e-11),
        # the analysis step: field and density of a 1,961-atom solution on a 64^3 grid
        dict(name='field_ag_1961_64', kind='field', shape='ag', size=20.0, grid=64),
    ]


def draw(rng):
    def spread(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    kind = rng.choice(['matvec', 'contract', 'plain', 'direct', 'mixed', 'fresh', 'otf', 'bowtie', 'bem', 'serve',
                       'field'])
    if kind == 'matvec':
        shape = rng.choice(['na', 'ag', 'bowtie'])
        size = {'na': rng.uniform(10.0, 32.0), 'ag': rng.uniform(7.0, 20.0), 'bowtie': rng.uniform(20.0, 45.0)}[shape]
        return dict(kind='matvec', shape=shape, size=round(size, 2), otf=rng.random() < 0.5)
    if kind == 'contract':
        shape = rng.choice(['na', 'ag'])
        size = rng.uniform(16.0, 40.0) if shape == 'na' else rng.uniform(9.0, 25.0)
        return dict(kind='contract', shape=shape, size=round(size, 2), count=int(round(spread(1, 48))))
    if kind == 'plain':
        shape = rng.choice(['na', 'ag'])
        size = rng.uniform(10.0, 24.0) if shape == 'na' else rng.uniform(7.0, 14.0)
        return dict(kind='solve', shape=shape, size=round(size, 2), n_freq=int(round(spread(5, 61))),
                    pol=rng.choice(['x', 'x', 'all']), mode='iterative', precision='fp64', inner=0, inner_tol=0.0,
                    rtol=1e-11, fresh=False)
    if kind == 'direct':
        return dict(kind='solve', shape='na', size=round(rng.uniform(9.0, 22.0), 2), n_freq=int(round(spread(5, 61))),
                    pol=rng.choice(['x', 'all']), mode='inversion', precision='fp64', inner=0, inner_tol=0.0,
                    rtol=0.0, fresh=True)
    if kind == 'mixed':
        p = rng.choice(['mixed_bf16x3', 'mixed_bf16'])
        return dict(kind='solve', shape='ag', size=round(rng.uniform(8.0, 21.0), 2), n_freq=int(round(spread(11, 81))),
                    pol='x', mode='iterative', precision=p, inner=64, inner_tol=1e-4 if p == 'mixed_bf16x3' else 3e-2,
                    rtol=2e-11, fresh=False)
    if kind == 'fresh':
        return dict(kind='solve', shape='ag', size=round(rng.uniform(18.0, 33.0), 2), n_freq=rng.randint(5, 21),
                    pol='x', mode='iterative', precision='mixed_bf16', inner=64, inner_tol=3e-2, rtol=2e-11,
                    fresh=True)
    if kind == 'otf':
        shape = rng.choice(['ag', 'bowtie'])
        size = rng.uniform(8.0, 13.0) if shape == 'ag' else rng.uniform(18.0, 29.0)
        return dict(kind='solve', shape=shape, size=round(size, 2), n_freq=rng.randint(1, 8), pol='x',
                    mode='iterative on the fly', precision='fp64', inner=0, inner_tol=0.0, rtol=1e-11, fresh=False)
    if kind == 'bowtie':
        return dict(kind='solve', shape='bowtie', size=round(rng.uniform(30.0, 58.0), 2), n_freq=rng.randint(7, 31),
                    pol='x', mode='iterative on the fly', precision='mixed_bf16x3', inner=256, inner_tol=1e-3,
                    rtol=2e-11, fresh=False)
    if kind == 'bem':
        return dict(kind='bem', shape=rng.choice(['sphere', 'rod']), n_tess=int(round(spread(500, 8000))),
                    n_freq=int(round(spread(21, 301))), pol=rng.choice(['x', 'z']),
                    precision=rng.choice(['mixed_bf16x3', 'mixed_bf16x3', 'fp64']), rtol=1e-11)
    if kind == 'serve':
        return dict(kind='serve', size=round(rng.uniform(9.0, 15.0), 2), requests=rng.randint(2, 8),
                    n_freq=int(round(spread(20, 60))), rtol=2e-11)
    shape = rng.choice(['na', 'ag'])
    return dict(kind='field', shape=shape, size=round(rng.uniform(9.0, 21.0), 2), grid=int(round(spread(15, 68))))


# ---- inputs -----------------------------------------------------------------


def _problem(case, seed, shape=None, size=None):
    """Geometry and frequency grid of an atomistic case."""
    shape = shape or case['shape']
    size = size or case['size']
    kw = dict(n_freq=case.get('n_freq', 3), seed=seed, jitter=JITTER, method=case.get('mode', 'iterative'),
              polarization=case.get('pol', 'x'))
    if shape == 'na':
        return configs.na_sphere(radius=size, **kw)
    if shape == 'ag':
        return configs.ag_sphere(radius=size, **kw)
    if shape == 'bowtie':
        return configs.agau_bowtie(edge=size, **kw)
    metal, form = shape.split('_')
    return configs.particle(metal, form, size, **kw)


# the geometries of a serving case, in turn: metal and form, and radius over the case's size
SERVED = [('Na_sphere', 1.25), ('Ag_sphere', 1.0), ('Au_rod', 0.55), ('Na_rod', 0.6), ('Au_sphere', 0.8),
          ('Ag_rod', 0.5), ('Na_sphere', 0.9), ('Ag_sphere', 0.75)]


def _served(case, seed):
    return [_problem(case, seed + 7919 * k, shape, case['size'] * scale)
            for k, (shape, scale) in enumerate(SERVED[:case['requests']])]


def _surface(case, seed):
    return bem.bem_surface(case['n_tess'], shape=case['shape'], n_freq=case['n_freq'], seed=seed,
                           polarization=case['pol'], method='iterative')


def _columns(n, count, seed):
    return np.random.default_rng(seed).standard_normal((count, n))


def _vector(n, seed):
    a = _columns(n, 2, seed)
    return a[0] + 1j * a[1]


def _points(prob, grid):
    """Points (bohr) of the analysis step's cubic grid around the particle."""
    return np.ascontiguousarray(analysis.cubic_grid(prob.coord_ang, (grid, grid, grid)).points_ang() * TO_BOHR)


class State:
    """What a program holds between calls; releases the geometries before their context."""

    def __init__(self, case):
        self.case = case
        self.solvers = []
        self.ctx = Context(0)

    def resident(self, prob, **kw):
        s = Solver(prob, ctx=self.ctx, **kw)
        self.solvers.append(s)
        return s

    def __del__(self):
        for s in self.solvers:
            s.close()
        self.ctx.close()


def _tol(solver, rtol, pol):
    b = solver.rhs(0, {'x': 1, 'y': 2, 'z': 4, 'all': 7}[pol])
    return rtol * float(np.linalg.norm(b, axis=0).max())


def prepare(case, seed):
    st = State(case)
    kind = case['kind']
    if kind == 'bem':
        st.solver = st.resident(_surface(case, seed))
        st.tol = _tol(st.solver, case['rtol'], case['pol'])
        return st
    if kind == 'serve':
        st.probs = _served(case, seed)
        for p in st.probs:
            st.resident(p, store_t=True)
        st.tols = [_tol(s, case['rtol'], 'x') for s in st.solvers]
        return st
    st.prob = _problem(case, seed)
    if kind == 'matvec':
        st.solver = st.resident(st.prob, store_t=not case['otf'])
        st.x = _vector(st.prob.n_var, seed)
    elif kind == 'contract':
        st.solver = st.resident(st.prob, store_t=True)
        st.x = _columns(st.prob.n_var, case['count'], seed)
    elif kind == 'field':
        st.solver = st.resident(st.prob, store_t=False)
        # charges and dipoles of the size a solution has (field intensity 1e-4)
        st.x = 1e-3 * _vector(st.prob.n_var, seed)
        st.points = _points(st.prob, case['grid'])
    elif case['fresh']:
        # the geometry is built in the pass; the tolerance comes from the field and size alone
        st.tol = _fresh_tol(case, st.prob)
    else:
        st.solver = st.resident(st.prob)
        st.tol = _tol(st.solver, case['rtol'], case['pol'])
    return st


def _fresh_tol(case, prob):
    """rtol times the norm the right-hand side of a silver particle has: its surface charge rows,
    about 22 E0 times the cube root of the number of atoms (zero for a direct solve)."""
    return case['rtol'] * 22.0 * prob.e0 * prob.n_atoms ** (1.0 / 3.0)


# ---- one pass ----------------------------------------------------------------


def _solve(st, solver):
    c = st.case
    out = solver.solve(precision=c['precision'], tol=st.tol, max_krylov=3000, inner_krylov=c['inner'],
                       inner_tol=c['inner_tol'])
    return {'results': out['results'], 'polar': out['polar'], 'status': out['status']}


def run(st):
    c = st.case
    kind = c['kind']
    if kind == 'matvec':
        return st.solver.matvec(1, st.x, on_the_fly=c['otf'])
    if kind == 'contract':
        return st.solver.contract(st.x, 'fp64')
    if kind == 'field':
        return st.solver.field_at_points(0, st.x, st.points)
    if kind == 'bem':
        out = st.solver.solve(precision=c['precision'], tol=st.tol)
        return {'results': out['results'], 'polar': out['polar'], 'status': out['status']}
    if kind == 'serve':
        return _serve(st)
    if c['fresh']:
        with Solver(st.prob, ctx=st.ctx) as solver:
            return _solve(st, solver)
    return _solve(st, st.solver)


def _serve(st):
    batches = [Batch(s, precision='mixed_bf16x3') for s in st.solvers]
    outs = {}
    try:
        for k, (b, p) in enumerate(zip(batches, st.probs)):
            b.add(k, p.freqs, p.alpha_w, pol_mask=1, tol=st.tols[k])
        while True:
            live = [b for b in batches if b.active]
            if not live:
                break
            Batch.step_group(live)
        for k, b in enumerate(batches):
            outs[k] = b.take(k)
    finally:
        for b in batches:
            b.close()
    return [{'results': outs[k]['results'], 'polar': outs[k]['polar'], 'status': outs[k]['status']}
            for k in range(len(batches))]


# ---- what a pass cannot do without -------------------------------------------

# sites per cubic Angstrom of the lattices and the volumes of the shapes
DENSITY = {'na': 2 / 4.225 ** 3, 'ag': 4 / 4.086 ** 3, 'au': 4 / 4.08 ** 3}


def _atoms(shape, size):
    if shape == 'bowtie':
        return int(DENSITY['au'] * 2 * 20.0 * math.sqrt(3) / 4 * size ** 2 * 1.1)
    metal, form = (shape.lower().split('_') + ['sphere'])[:2]
    vol = 4 / 3 * math.pi * size ** 3 + (2 * math.pi * size ** 3 if form == 'rod' else 0.0)
    return int(DENSITY[metal] * vol)


# Arnoldi steps a column takes at the tolerances above (the order of what is measured)
STEPS = {'na': 130, 'ag': 250, 'au': 200, 'bowtie': 500, 'sphere': 20, 'rod': 80}


def _spectrum_work(n, atoms, cols, steps, build):
    # each Arnoldi step multiplies T by the real and imaginary part of every column; a fresh
    # geometry evaluates every pair of atoms once (a few hundred operations)
    return {'bytes': 8.0 * n * n + 16.0 * n * cols, 'flops': 4.0 * n * n * cols * steps + (200.0 * atoms ** 2 if build else 0.0)}


def work(case):
    kind = case['kind']
    if kind == 'bem':
        n = 20 * max(1, round(math.sqrt(case['n_tess'] / 20.0))) ** 2
        return _spectrum_work(n, n, case['n_freq'], STEPS[case['shape']], False)
    if kind == 'serve':
        w = {'bytes': 0.0, 'flops': 0.0}
        for shape, scale in SERVED[:case['requests']]:
            atoms = _atoms(shape, case['size'] * scale)
            metal = shape.split('_')[0].lower()
            one = _spectrum_work(atoms if metal == 'na' else 4 * atoms, atoms, case['n_freq'], STEPS[metal], False)
            w = {k: w[k] + one[k] for k in w}
        return w
    shape, atoms = case['shape'], _atoms(case['shape'], case['size'])
    n = atoms if shape == 'na' else 4 * atoms
    if kind == 'matvec':
        if case['otf']:
            # every pair of atoms: its 16 (1) elements and the products
            return {'bytes': 32.0 * n + 64.0 * atoms, 'flops': (400.0 if n > atoms else 60.0) * atoms ** 2}
        return {'bytes': 8.0 * n * n + 32.0 * n, 'flops': 4.0 * n * n}
    if kind == 'contract':
        return {'bytes': 8.0 * n * n + 16.0 * n * case['count'], 'flops': 2.0 * n * n * case['count']}
    if kind == 'field':
        pts = case['grid'] ** 3
        return {'bytes': 16.0 * n + 40.0 * atoms + 88.0 * pts, 'flops': (150.0 if n > atoms else 60.0) * atoms * pts}
    cols = case['n_freq'] * (3 if case['pol'] == 'all' else 1)
    if case['mode'] == 'inversion':
        # one reduction of the real matrix, then O(n^2) a column
        return {'bytes': 8.0 * n * n + 16.0 * n * cols, 'flops': 10 / 3 * n ** 3 + 24.0 * n * n * cols + 200.0 * atoms ** 2}
    return _spectrum_work(n, atoms, cols, STEPS[shape], case['fresh'])


# ---- the same outputs from plain torch in 64 bits ------------------------------


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a), device='cuda')


def _pair_geometry(p):
    r = _dev(p.coord)
    d = r[:, None, :] - r[None, :, :]
    r2 = (d * d).sum(-1)
    r2.fill_diagonal_(1.0)
    return d, r2.sqrt()


def _damp(r, R):
    u = r / R
    e = torch.exp(-u * u)
    return torch.erf(u) - 2.0 / math.sqrt(math.pi) * u * e, e


def _interaction(p):
    """T: charges, then dipoles x, y, z of every atom in turn."""
    N = p.n_atoms
    t = _dev(p.atom_types).long()
    d, r = _pair_geometry(p)
    rq = _dev(p.r_q)[t]
    qq = torch.erf(r / (rq[:, None] ** 2 + rq[None, :] ** 2).sqrt()) / r
    qq.diagonal().copy_(_dev(p.eta)[t])
    if p.model == 'wfq':
        return qq
    rm = _dev(p.r_mu)[t]
    T = torch.zeros(4 * N, 4 * N, dtype=torch.float64, device='cuda')
    T[:N, :N] = qq
    del qq
    f, _ = _damp(r, (rq[:, None] ** 2 + rm[None, :] ** 2).sqrt())
    f = f / r ** 3
    f.fill_diagonal_(0.0)
    for k in range(3):
        T[:N, N + k::3] = d[:, :, k] * f
        T[N + k::3, :N] = T[:N, N + k::3].T
    R = (rm[:, None] ** 2 + rm[None, :] ** 2).sqrt()
    f1, e = _damp(r, R)
    f2 = 4.0 / (math.sqrt(math.pi) * R ** 3) * e
    a = -3.0 * f1 / r ** 5 + f2 / r ** 2
    b = f1 / r ** 3
    a.fill_diagonal_(0.0)
    b.fill_diagonal_(0.0)
    for k in range(3):
        for m in range(3):
            T[N + k::3, N + m::3] = a * d[:, :, k] * d[:, :, m] + (b if k == m else 0.0)
    return T


def _conductance(p):
    t = _dev(p.atom_types).long()
    _, r = _pair_geometry(p)
    pair = lambda m: _dev(m)[t[:, None], t[None, :]]  # noqa: E731
    K = torch.sigmoid(-pair(p.fermi_d) * (r / (pair(p.fermi_s) * pair(p.r0)) - 1.0))
    K = K * _dev(p.a_ij)[t][:, None] / r
    # the model's factor is 1 - 1 / (1 + exp(-u)): zero where that rounds to zero
    u = pair(p.fermi_d) * (r / (pair(p.fermi_s) * pair(p.r0)) - 1.0)
    K[(1.0 - 1.0 / (1.0 + torch.exp(-u))) == 0.0] = 0.0
    K.fill_diagonal_(0.0)
    return K


def _charge_operator(p, K, w):
    """Kop(w): rows sum_j c_ij (s_j - s_i)."""
    if len(p.type_names) == 1:
        c = K
    else:
        t = _dev(p.atom_types).long()
        wt = _dev(2.0 * p.density / (1.0 / p.tau - 1j * w))[t]
        c = 0.5 * (K + wt[None, :] / wt[:, None] * K.T)
    return c - torch.diag(c.sum(1))


def _diagonal(p, w, i):
    t = p.atom_types
    z = w * (-w * p.tau - 1j) / (2.0 * p.density * p.tau)
    dq = -z[t]
    if p.model == 'wfq':
        return _dev(dq)
    if len(p.type_names) > 1:
        raise ValueError('dipole diagonal of an alloy needs its neighbour fractions')
    return _dev(np.concatenate([dq, np.repeat(1.0 / p.alpha_w[t, i], 3)]))


def _alloy_diagonal(p, w, i, frac):
    z = w * (-w * p.tau - 1j) / (2.0 * p.density * p.tau)
    ia = (frac * (1.0 / p.alpha_w[:, i])[:, None]).sum(0)
    return _dev(np.concatenate([-z[p.atom_types], np.repeat(ia, 3)]))


def _fractions(p):
    """Share of each atom's neighbours (itself included) that are of each type; counted from
    the Angstrom coordinates, an atom of another element in its own type."""
    nt = len(p.type_names)
    xyz = p.coord_ang
    nb = np.zeros((nt, p.n_atoms))
    for i in range(p.n_atoms):
        d = np.sqrt(((xyz - xyz[i]) ** 2).sum(1)) * TO_BOHR
        hit = d <= p.r0[p.atom_types[i], p.atom_types]
        hit[i] = True
        nb[:, i] = np.bincount(p.atom_types[hit], minlength=nt)
    return nb / nb.sum(0)


def _rhs(p, kop, pol):
    N = p.n_atoms
    v = _dev(-p.e0 * p.coord[:, pol])
    b = -(kop @ v.to(kop.dtype))
    if p.model == 'wfq':
        return b
    m = torch.zeros(3 * N, dtype=kop.dtype, device='cuda')
    m[pol::3] = p.e0
    return torch.cat([b, m])


def _row(P, w):
    """The 20 results of a frequency from its 3 x 3 polarizability."""
    iso = np.trace(P) / 3
    d = np.diag(P)
    al = np.concatenate([[iso], d])
    ab = 4 * math.pi * w * al.imag / LIGHT
    sc = 8 * math.pi * w ** 4 * np.abs(al) ** 2 / (3 * LIGHT ** 4)
    return np.concatenate([[iso.real, iso.imag], d.real, d.imag, ab, sc, ab + sc])


def _spectrum(p, pols, A_of, b_of, weight, dipoles):
    F = len(p.freqs)
    polar = np.zeros((F, 3, 3), dtype=np.complex128)
    res = np.zeros((F, 20))
    for i, w in enumerate(p.freqs):
        A, bs = A_of(i), b_of(i)
        x = torch.linalg.solve(A, torch.stack(bs, 1)).cpu().numpy()
        for c, pol in enumerate(pols):
            q = x[:len(weight), c]
            for a in range(3):
                polar[i, a, pol] = (q * weight[:, a]).sum() / p.e0
                if dipoles:
                    polar[i, a, pol] += x[len(weight) + a::3, c].sum() / p.e0
        res[i] = _row(polar[i], w)
    return {'results': res, 'polar': polar, 'status': None}


def _exact_spectrum(p, pol):
    pols = {'x': [0], 'y': [1], 'z': [2], 'all': [0, 1, 2]}[pol]
    N = p.n_atoms
    T, K = _interaction(p), _conductance(p)
    alloy = len(p.type_names) > 1
    frac = _fractions(p) if alloy else None
    if not alloy:
        kop = _charge_operator(p, K, 0.0)
        A0 = T.clone()
        A0[:N] = kop @ T[:N]
        b0 = [_rhs(p, kop, c).to(torch.complex128) for c in pols]

    def operator(i):
        if not alloy:
            A = A0.to(torch.complex128)
            A.diagonal().add_(_diagonal(p, p.freqs[i], i))
            return A
        k = _charge_operator(p, K, p.freqs[i])
        A = T.to(torch.complex128)
        A[:N] = torch.complex(k.real @ T[:N], k.imag @ T[:N])
        A.diagonal().add_(_alloy_diagonal(p, p.freqs[i], i, frac))
        return A

    def rhs(i):
        if not alloy:
            return b0
        k = _charge_operator(p, K, p.freqs[i])
        return [_rhs(p, k, c) for c in pols]

    return _spectrum(p, pols, operator, rhs, p.coord, p.model == 'wfqfmu')


def _exact_bem(case, p):
    tri = _dev(p.triangles)
    c = tri.mean(1)
    cr = torch.linalg.cross(tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0])
    nc = cr.norm(dim=1)
    nrm, area = p.normal_factor * cr / nc[:, None], nc / 2
    d = c[:, None, :] - c[None, :, :]
    r = d.norm(dim=2)
    r.fill_diagonal_(1.0)
    D = area[None, :] * (d * nrm[:, None, :]).sum(2) / r ** 3
    D.diagonal().copy_(1.0694 * (4 * math.pi * area).sqrt() / (2 * p.sphere_radius))
    del d, r
    z = 2 * math.pi * (p.eps_solvent + p.eps) / (p.eps_solvent - p.eps)
    pol = 'xyz'.index(case['pol'])
    b = (-p.e0 * nrm[:, pol]).to(torch.complex128)
    D = D.to(torch.complex128)

    def operator(i):
        A = D.clone()
        A.diagonal().add_(complex(z[i]))
        return A

    return _spectrum(p, [pol], operator, lambda i: [b], (c * area[:, None]).cpu().numpy(), False)


def _exact_field(p, x, pts):
    """E0 plus the field of charges and dipoles, and the density, at every point, for a block of
    points at a time."""
    N = p.n_atoms
    r_at, P = _dev(p.coord), _dev(pts)
    q = _dev(x[:N])
    rq = _dev(p.r_q)[_dev(p.atom_types).long()]
    fmu = p.model == 'wfqfmu'
    if fmu:
        mu = _dev(x[N:]).reshape(N, 3)
        rm = _dev(p.r_mu)[_dev(p.atom_types).long()]
    E = torch.zeros(len(pts), 3, dtype=torch.complex128, device='cuda')
    rho = torch.zeros(len(pts), dtype=torch.complex128, device='cuda')
    step = max(1, int(1.0e7 // N))
    p32 = math.pi ** 1.5
    cx = lambda a: a.to(torch.complex128)  # noqa: E731
    for k in range(0, len(pts), step):
        d = r_at[None, :, :] - P[k:k + step, None, :]
        r = d.norm(dim=2)
        far = r > 0.1
        s = torch.where(far, r, torch.ones_like(r))
        eq = torch.exp(-(r / rq) ** 2)
        f = torch.where(far, (torch.erf(r / rq) - 2 / math.sqrt(math.pi) / rq * r * eq) / s ** 3, 0.0)
        E[k:k + step] = -torch.einsum('pnk,n->pk', cx(d * f[:, :, None]), q)
        rho[k:k + step] = cx(eq / (p32 * rq ** 3)) @ q
        if fmu:
            em = torch.exp(-(r / rm) ** 2)
            f1 = torch.erf(r / rm) - 2 / math.sqrt(math.pi) / rm * r * em
            f2 = 4 / (math.sqrt(math.pi) * rm ** 3) * em
            a = torch.where(far, -3 * f1 / s ** 5 + f2 / s ** 2, 0.0)
            b = torch.where(far, f1 / s ** 3, 0.0)
            dm = torch.einsum('pnk,nk->pn', cx(d), mu)
            E[k:k + step] += torch.einsum('pnk,pn->pk', cx(d * a[:, :, None]), dm) + cx(b) @ mu
            rho[k:k + step] -= (2 * em / (p32 * rm ** 5) * dm).sum(1)
    E[:, 0] += p.e0
    return E.cpu().numpy(), rho.cpu().numpy()


def exact(case, seed):
    kind = case['kind']
    if kind == 'bem':
        return _exact_bem(case, _surface(case, seed))
    if kind == 'serve':
        return [_exact_spectrum(p, 'x') for p in _served(case, seed)]
    p = _problem(case, seed)
    if p.n_var > 16000:
        return _exact_contract(p, case, seed) if kind == 'contract' else None
    if kind == 'contract':
        return _exact_contract(p, case, seed)
    if kind == 'matvec':
        x = _vector(p.n_var, seed)
        v = _dev(x)
        T, w = _interaction(p), p.freqs[1]
        s = torch.complex(T @ v.real, T @ v.imag)
        N = p.n_atoms
        kop = _charge_operator(p, _conductance(p), w)
        y = s.clone()
        y[:N] = kop.to(torch.complex128) @ s[:N]
        y += (_alloy_diagonal(p, w, 1, _fractions(p)) if len(p.type_names) > 1 else _diagonal(p, w, 1)) * v
        return y.cpu().numpy()
    if kind == 'field':
        return _exact_field(p, 1e-3 * _vector(p.n_var, seed), _points(p, case['grid']))
    return _exact_spectrum(p, case['pol'])


def _exact_contract(p, case, seed):
    return (_dev(_columns(p.n_var, case['count'], seed)) @ _interaction(p)).cpu().numpy()
