"""Performance cases: the device work that a program using this package repeats.

A case names an operation, a molecule, a Becke grid (nrad x nang points per
atom) and a precision; ``prepare`` builds what a program holds between calls
(grid, basis, Fock plan, inputs on the device) and ``run`` makes one pass
through the public entry points.  ``exact`` gives the same results in 64-bit
torch, written from the formulas: contracted Cartesian Gaussians, Becke's
weights, the density and the quadrature as matrix products, and the
Becke-Dickson Poisson solve (Lebedev projection, radial equation by cubic
Hermite finite elements, multipole evaluation).  It takes only published data
from the package: element radii, basis sets and the Lebedev rules.
"""
import math

import numpy as np
import torch

import napmo_b200 as nb
from napmo_b200.gradients import GridChargeEnergy
from napmo_b200.grids import ELEMENTS
from napmo_b200.gto import shells_for
from napmo_b200.scf import GridRHF
from napmo_b200.system import (BOHR_TO_ANGSTROM, alkane_geometry, build_system, h2o_geometry,
                               hcn_geometry, random_batch)

BASIS = 'CC-PVDZ'
SMALL_RULES = (50, 74, 86, 110, 146, 170, 194)
RULES = (110, 146, 170, 194, 230, 266, 302, 350)


def listed():
    return [
        # the density of a small molecule, once per SCF iteration: launches and latency
        dict(name='density_h2o', op='density', molecule='H2O', nrad=50, nang=110,
             precision='fp64'),
        # the density of a mid-size molecule on the tensor cores
        dict(name='density_c8h18_int8', op='density', molecule='C8', nrad=100, nang=302,
             precision='int8x4'),
        # one quadrature of a potential (nuclear attraction, coupling, XC matrix)
        dict(name='quadrature_c8h18', op='quadrature', molecule='C8', nrad=100, nang=302,
             precision='fp64'),
        # one Coulomb potential, on the grid of the gradient workload
        dict(name='potential_c5h12', op='potential', molecule='C5', nrad=75, nang=194,
             precision='fp64'),
        # the pair densities of one occupied orbital: the exchange part of an SCF step
        dict(name='potentials_hcn', op='potentials', molecule='HCN', nrad=100, nang=302,
             precision='fp64', solves=35),
        # whole Fock builds: the smallest, an FP64 one, and the largest system with
        # its contractions on the tensor cores
        dict(name='build_h2o', op='build', molecule='H2O', nrad=50, nang=110,
             precision='fp64'),
        dict(name='build_c12h26', op='build', molecule='C12', nrad=100, nang=302,
             precision='fp64'),
        dict(name='build_c20h42_int8', op='build', molecule='C20', nrad=100, nang=302,
             precision='int8x4'),
        # the Hartree-Fock exchange matrix of one SCF iteration
        dict(name='exchange_h2o_int8', op='exchange', molecule='H2O', nrad=50, nang=110,
             precision='int8x4'),
        # many molecules of uneven basis and grid sizes in one launch
        dict(name='batch_8_int8', op='batch', molecule='chains', count=8, geometry=20261203,
             mode='stages', precision='int8x4'),
        # energy and its derivatives (forward and backward) at two geometries
        dict(name='gradient_h2o', op='gradient', molecule='H2O', nrad=75, nang=194,
             precision='fp64'),
        # one geometry step of a Fock plan: weights, basis values, Poisson tables
        dict(name='move_c4h10', op='move', molecule='C4', nrad=75, nang=194,
             precision='fp64'),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(('density', 'quadrature', 'potential', 'potentials', 'build', 'exchange',
                     'batch', 'gradient', 'move'))
    precision = rng.choice(('fp64', 'int8x4'))
    if op == 'batch':
        return dict(op=op, molecule='chains', count=rng.randint(2, 6),
                    geometry=rng.randrange(1 << 20), mode=rng.choice(('streams', 'stages')),
                    precision=precision)
    if op in ('potentials', 'exchange', 'gradient'):
        case = dict(op=op, molecule=rng.choice(('H2O', 'HCN', 'C1')), nrad=rng.randint(30, 80),
                    nang=rng.choice(SMALL_RULES), precision=precision)
        if op == 'potentials':
            case['solves'] = _log_int(rng, 2, 60)
        return case
    most = {'move': 6, 'build': 12, 'potential': 12}.get(op, 16)
    molecule = rng.choice(('H2O', 'HCN') + ('C%d' % _log_int(rng, 1, most),) * 3)
    return dict(op=op, molecule=molecule, nrad=rng.randint(30, 100), nang=rng.choice(RULES),
                precision=precision)


# ------------------------------------------------------------------ molecules
def _atoms(molecule):
    """[(symbol, xyz in angstrom)]; 'Cn' is the all-trans alkane of n carbons."""
    if molecule == 'H2O':
        return h2o_geometry()
    if molecule == 'HCN':
        return hcn_geometry()
    return alkane_geometry(int(molecule[1:]))


def _molecules(case):
    """[(atoms, nrad per atom, nang per atom)] of a case."""
    if case['op'] == 'batch':
        return [(m['atoms'], m['nrad'], m['nang'])
                for m in random_batch(case['count'], case['geometry'], natom=(3, 20))]
    atoms = _atoms(case['molecule'])
    return [(atoms, [case['nrad']] * len(atoms), [case['nang']] * len(atoms))]


def _functions(symbol):
    return sum((l + 1) * (l + 2) // 2 for l, _, _ in shells_for(BASIS, symbol))


def _bohr(atoms):
    return np.array([xyz for _, xyz in atoms]) / BOHR_TO_ANGSTROM


def _electrons(atoms):
    return sum(ELEMENTS[s]['atomic_number'] for s, _ in atoms)


# --------------------------------------------------------------------- inputs
def _generator(seed, k=0):
    return torch.Generator().manual_seed(1000003 * seed + k)


def _density_matrix(n, nocc, seed, k=0):
    """2 C C^T of normal coefficients, n x nocc."""
    C = torch.randn(n, nocc, dtype=torch.float64, generator=_generator(seed, k)) / math.sqrt(n)
    return (2.0 * C @ C.T).cuda()


def _potential(points, centers, seed):
    """Potential of a smeared charge on every centre (charges near 4)."""
    q = 4.0 + torch.randn(len(centers), dtype=torch.float64, generator=_generator(seed))
    v = torch.zeros(points.shape[0], dtype=torch.float64, device='cuda')
    for a, R in enumerate(centers):
        d = (points - R).norm(dim=1)
        v -= q[a].item() * torch.erf(1.3 * d) / d
    return v


def _charge_density(points, centers, charges, seed):
    """An exponential density on every centre with a dipolar distortion."""
    p = torch.randn(len(centers), 3, dtype=torch.float64, generator=_generator(seed)).cuda()
    rho = torch.zeros(points.shape[0], dtype=torch.float64, device='cuda')
    for a, R in enumerate(centers):
        x = points - R
        d = x.norm(dim=1)
        rho += charges[a] * torch.exp(-1.7 * d) * (1.0 + 0.2 * (x @ p[a]) / (1.0 + d))
    return rho


def _orbitals(case, seed):
    """Occupied orbital coefficients (n x nocc, orthonormal columns)."""
    atoms = _atoms(case['molecule'])
    n = sum(_functions(s) for s, _ in atoms)
    C = torch.randn(n, _electrons(atoms) // 2, dtype=torch.float64, generator=_generator(seed))
    return torch.linalg.qr(C)[0].cuda()


def _pair_densities(case, phi, seed):
    """psi phi_nu of one random orbital with `solves` basis functions."""
    n = phi.shape[0]
    c = torch.randn(n, dtype=torch.float64, generator=_generator(seed)).cuda() / math.sqrt(n)
    rows = [k % n for k in range(case['solves'])]
    return (c @ phi) * phi[rows]


def _displaced(case, seed, k):
    """Atom positions (bohr) moved by 0.02 bohr normal displacements."""
    R = torch.as_tensor(_bohr(_atoms(case['molecule'])))
    return R + 0.02 * torch.randn(R.shape, dtype=torch.float64, generator=_generator(seed, k))


def _symbols(case):
    return [s for s, _ in _atoms(case['molecule'])]


# ------------------------------------------------------------- prepare and run
def _builder(atoms, nrad, nang, precision):
    ms = build_system(atoms, BASIS)
    uneven = len(set(nrad)) > 1 or len(set(nang)) > 1
    grid = nb.BeckeGrid(ms['e-'], nrad if uneven else nrad[0], nang if uneven else nang[0])
    lmax = 'per-atom' if uneven else nb.lebedev_get_order(nang[0]) // 2
    return grid, ms['e-']['basis'], nb.FockBuilder(grid, ms['e-']['basis'], lmax,
                                                   precision=precision)


def prepare(case, seed):
    op, precision = case['op'], case['precision']
    mols = _molecules(case)
    if op == 'batch':
        builders = [_builder(*m, precision)[2] for m in mols]
        batch = nb.FockBatch(builders)
        batch.set_mode(case['mode'])
        for k, (b, m) in enumerate(zip(builders, mols)):
            batch.D(k).copy_(_density_matrix(b.n, max(1, _electrons(m[0]) // 2), seed, k))
        return dict(op=op, batch=batch)
    atoms = mols[0][0]
    centers = torch.as_tensor(_bohr(atoms)).cuda()
    if op == 'gradient':
        model = GridChargeEnergy(_symbols(case), basis=BASIS, nrad=case['nrad'],
                                 nang=case['nang'], precision=precision)
        n = sum(_functions(s) for s in _symbols(case))
        D = _density_matrix(n, _electrons(atoms) // 2, seed)
        return dict(op=op, model=model, D=D, R=[_displaced(case, seed, k) for k in (1, 2)])
    if op == 'exchange':
        scf = GridRHF(build_system(atoms, BASIS), case['nrad'], case['nang'],
                      precision=precision)
        return dict(op=op, scf=scf, C=_orbitals(case, seed))
    grid, basis, plan = _builder(*mols[0], precision)
    state = dict(op=op, grid=grid, basis=basis, plan=plan)
    if op in ('density', 'build'):
        state['D'] = _density_matrix(plan.n, _electrons(atoms) // 2, seed)
    elif op == 'move':
        R = _displaced(case, seed, 1).numpy()
        origins = basis.origins()
        of = [int(np.argmin(((_bohr(atoms) - o) ** 2).sum(1))) for o in origins]
        state['centers'], state['origins'] = R, R[of]
    else:
        points = torch.as_tensor(grid.points.copy()).cuda()
        if op == 'quadrature':
            state['v'] = _potential(points, centers, seed)
        elif op == 'potential':
            charges = [ELEMENTS[s]['atomic_number'] for s, _ in atoms]
            state['rho'] = _charge_density(points, centers, charges, seed)
        else:
            state['rho'] = _pair_densities(case, _basis_values(_symbols(case), centers, points),
                                           seed)
    return state


def run(state):
    op = state['op']
    if op == 'batch':
        return [F.clone() for F in state['batch'].build()]  # the batch's own buffers
    if op == 'gradient':
        out = []
        for R in state['R']:
            D = state['D'].clone().requires_grad_(True)
            R = R.clone().requires_grad_(True)
            E = state['model'](D, R)
            E.backward()
            out.append((E.detach(), D.grad, R.grad))
        return out
    if op == 'exchange':
        return state['scf'].exchange_matrix(state['C'])
    plan = state['plan']
    if op == 'density':
        return plan.density(state['D'])
    if op == 'quadrature':
        return plan.quadrature(1.0, state['v'])
    if op == 'potential':
        return plan.coulomb_potential(state['rho'])
    if op == 'potentials':
        return plan.coulomb_potentials(state['rho'])
    if op == 'move':
        state['grid'].set_centers(state['centers'])
        state['basis'].set_origins(state['origins'])
        plan.refresh()
        # copies: both are views of buffers that go with the grid and the plan
        return state['grid'].becke_weights.copy(), plan.phi()[:, :plan.npoint].clone()
    return plan.build(state['D'])


def work(case):
    """Least bytes and floating point operations of one pass: every input read
    once and every output written once; symmetric products by their upper
    triangle; per (atom, point) pair of a potential one product and sum for
    each cubic coefficient of its (lmax + 1)^2 multipoles."""
    nbytes = flops = 0.0
    for atoms, nrad, nang in _molecules(case):
        n = sum(_functions(s) for s, _ in atoms)
        N = sum(a * b for a, b in zip(nrad, nang))
        ls = [(nb.lebedev_get_order(a) // 2 + 1) ** 2 for a in nang]
        phi = 8.0 * n * N if case['precision'] == 'fp64' else 4.0 * n * N
        product = float(n) * (n + 1) * N
        project = sum(2.0 * a * b * l for a, b, l in zip(nrad, nang, ls))
        poisson = project + 8.0 * N * sum(ls)
        op = case['op']
        if op in ('density', 'quadrature'):
            nbytes += phi + 8.0 * (n * n + N)
            flops += product
        elif op == 'potential':
            nbytes += 16.0 * N
            flops += poisson
        elif op == 'potentials':
            nbytes += 16.0 * N * case['solves']
            flops += poisson * case['solves']
        elif op in ('build', 'batch'):
            nbytes += phi + 8.0 * (2 * n * n + (2 * N if op == 'build' else 0))
            flops += 2 * product + poisson
        elif op == 'exchange':
            k = n * (_electrons(atoms) // 2)
            nbytes += phi + 8.0 * n * n
            flops += k * poisson + 2.0 * k * N + product
        elif op == 'gradient':
            nbytes += 2 * (8.0 * 3 * N + 8.0 * 2 * n * n)
            flops += 2 * (3 * product + 30.0 * N * len(atoms) ** 2)
        else:
            nbytes += 8.0 * n * N + 8.0 * 4 * N
            flops += 15.0 * N * len(atoms) ** 2 + 10.0 * n * N
    return dict(bytes=nbytes, flops=flops)


# ----------------------------------------------------- results in 64-bit torch
def _norm(l, zeta, coef):
    """Contraction coefficients x primitive norms x the norm of their sum."""
    def odd(k):
        return math.prod(range(2 * k - 1, 0, -2))
    dd = odd(l[0]) * odd(l[1]) * odd(l[2])
    L = sum(l)
    z, c = np.asarray(zeta, dtype=np.float64), np.asarray(coef, dtype=np.float64)
    c = c * (2 * z / np.pi) ** 0.75 * (4 * z) ** (L / 2.0) / math.sqrt(dd)
    s = z[:, None] + z[None, :]
    S = (np.pi / s) ** 1.5 * dd / (2 * s) ** L
    return c / math.sqrt(c @ S @ c)


def _basis_values(symbols, centers, points):
    """phi [n][npoint] of the Cartesian contracted Gaussians at the points."""
    out = []
    for sym, R in zip(symbols, centers):
        x = points - R
        r2 = (x * x).sum(dim=1)
        for lval, zeta, coef in shells_for(BASIS, sym):
            e = [torch.exp(-z * r2) for z in zeta]
            for k in range(lval + 1):
                for j in range(k + 1):
                    l = (lval - k, k - j, j)
                    c = _norm(l, zeta, coef)
                    f = sum(c[i] * e[i] for i in range(len(zeta)))
                    for d in range(3):
                        if l[d]:
                            f = f * x[:, d] ** l[d]
                    out.append(f)
    return torch.stack(out)


def _becke(points, centers, radii, owner):
    """Becke's weight of every point for its owner (J. Chem. Phys. 88, 2547)."""
    nc = len(centers)
    if nc == 1:
        return torch.ones(points.shape[0], dtype=torch.float64, device='cuda')
    rad = torch.tensor(radii, dtype=torch.float64, device='cuda')
    chi = (rad[:, None] - rad[None, :]) / (rad[:, None] + rad[None, :])
    a = (chi / (chi * chi - 1.0)).clamp(-0.45, 0.45)
    off = ~torch.eye(nc, dtype=torch.bool, device='cuda')
    Rij = torch.where(off, (centers[:, None] - centers[None, :] + (~off)[..., None]).norm(dim=2),
                      torch.ones_like(chi))
    out = []
    step = max(1, (1 << 25) // (nc * nc))
    for i in range(0, points.shape[0], step):
        r = (points[i:i + step, None] - centers[None]).norm(dim=2)
        mu = (r[:, :, None] - r[:, None, :]) / Rij
        f = mu + a * (1.0 - mu * mu)
        for _ in range(3):
            f = 0.5 * f * (3.0 - f * f)
        P = torch.where(off, 0.5 * (1.0 - f), torch.ones_like(f)).prod(dim=2)
        own = owner[i:i + step]
        out.append(P[torch.arange(len(own), device='cuda'), own] / P.sum(dim=1))
    return torch.cat(out)


class _Atom(object):
    """Chebyshev radial grid r = R cot^2(theta / 2), theta = (n - t) pi / (n + 1),
    times a Lebedev rule; derivatives of r with respect to t."""

    def __init__(self, symbol, nrad, nang):
        self.R = ELEMENTS[symbol]['atomic_radii']
        self.n, self.nang = nrad, nang
        self.z = math.pi / (nrad + 1)
        theta = (nrad - torch.arange(nrad, dtype=torch.float64, device='cuda')) * self.z
        c = 1.0 / torch.tan(theta / 2)
        self.r = self.R * c * c
        self.j1 = self.z * self.R * c * (1 + c * c)
        self.j2 = self.z ** 2 * 0.5 * self.R * (1 + 3 * c * c) * (1 + c * c)
        self.j3 = self.z ** 3 * self.R * (2 * c + 3 * c ** 3) * (1 + c * c)
        self.w = 4 * math.pi * self.r * self.r * self.j1
        rule = nb.AngularGrid(nang)
        self.u = torch.as_tensor(rule.points.copy()).cuda()
        self.wang = torch.as_tensor(rule.weights.copy()).cuda()
        self.lmax = nb.lebedev_get_order(nang) // 2

    def points(self):
        return (self.r[:, None, None] * self.u[None]).reshape(-1, 3)

    def weights(self):
        return (self.w[:, None] * self.wang[None]).reshape(-1)


class _Grid(object):
    def __init__(self, atoms, nrad, nang, centers=None):
        self.symbols = [s for s, _ in atoms]
        self.centers = torch.as_tensor(_bohr(atoms)).cuda() if centers is None else centers
        self.atoms = [_Atom(s, a, b) for s, a, b in zip(self.symbols, nrad, nang)]
        self.size = [a.n * a.nang for a in self.atoms]
        self.points = torch.cat([a.points() + R for a, R in zip(self.atoms, self.centers)])
        self.w = torch.cat([a.weights() for a in self.atoms])
        self.owner = torch.cat([torch.full((s,), k, dtype=torch.long, device='cuda')
                                for k, s in enumerate(self.size)])
        self.becke = _becke(self.points, self.centers, [a.R for a in self.atoms], self.owner)

    def phi(self):
        return _basis_values(self.symbols, self.centers, self.points)


def _harmonics(x, lmax):
    """Real solid harmonics (sum over m of squares = 1) of unit vectors."""
    S = [None] * (lmax + 1) ** 2
    z = x[:, 2]
    c, s = torch.ones_like(z), torch.zeros_like(z)
    diag = 1.0
    for m in range(lmax + 1):
        if m:
            c, s = c * x[:, 0] - s * x[:, 1], c * x[:, 1] + s * x[:, 0]
            diag *= 1.0 if m == 1 else math.sqrt((2 * m - 1) / (2.0 * m))
        q, qp = torch.full_like(z, diag), torch.zeros_like(z)
        for l in range(m, lmax + 1):
            if l > m:
                a = (2 * l - 1) / math.sqrt(l * l - m * m)
                b = math.sqrt(((l - 1) ** 2 - m * m) / float(l * l - m * m))
                q, qp = a * z * q - b * qp, q
            if m == 0:
                S[l * l] = q
            else:
                S[l * l + 2 * m - 1] = q * c
                S[l * l + 2 * m] = q * s
    return torch.stack(S, dim=1)


def _spline(y):
    """t-derivatives of the natural cubic splines through the columns of y."""
    n = y.shape[0]
    M = torch.zeros(n, n, dtype=torch.float64, device='cuda')
    i = torch.arange(n, device='cuda')
    M[i, i] = 4.0
    M[0, 0] = M[-1, -1] = 2.0
    M[i[:-1], i[1:]] = M[i[1:], i[:-1]] = 1.0
    rhs = torch.empty_like(y)
    rhs[1:-1] = 3 * (y[2:] - y[:-2])
    rhs[0], rhs[-1] = 3 * (y[1] - y[0]), 3 * (y[-1] - y[-2])
    return torch.linalg.solve(M, rhs)


def _elements():
    """Integrals over one element of products of the four cubic Hermite
    functions H and their derivatives G: HH, GG, H G H, H H H."""
    x, w = np.polynomial.legendre.leggauss(6)
    x, w = 0.5 * (x + 1), 0.5 * w
    H = np.array([1 - 3 * x ** 2 + 2 * x ** 3, x - 2 * x ** 2 + x ** 3,
                  3 * x ** 2 - 2 * x ** 3, x ** 3 - x ** 2])
    G = np.array([6 * x ** 2 - 6 * x, 1 - 4 * x + 3 * x ** 2, 6 * x - 6 * x ** 2,
                  3 * x ** 2 - 2 * x])
    ein = (('ap,bp,p->ab', H, H), ('ap,bp,p->ab', G, G), ('ap,bp,cp,p->abc', H, G, H),
           ('ap,bp,cp,p->abc', H, H, H))
    return [torch.as_tensor(np.einsum(*e, w)).cuda() for e in ein]


def _radial_matrices(at):
    """Galerkin matrices [lmax + 1][2n][2n] of u'' + 2/r u' - l(l+1)/r^2 u on
    the t-axis, end values prescribed, and the source matrix [2n][2n]; the
    coefficient functions are their Hermite interpolants."""
    n, r, j1, j2, j3 = at.n, at.r, at.j1, at.j2, at.j3
    HH, GG, HGH, HHH = _elements()
    b = torch.stack([j1 * 2 / r - j2 / j1,
                     j2 * 2 / r - 2 * j1 * j1 / (r * r) + (j2 * j2 - j1 * j3) / (j1 * j1)], 1)
    a = torch.stack([-(j1 / r) ** 2, (2 * j1 * j1 / r ** 3 - 2 * j2 / (r * r)) * j1], 1)
    node = torch.arange(n - 1, device='cuda')
    dof = torch.stack([2 * node, 2 * node + 1, 2 * node + 2, 2 * node + 3], 1)
    be = torch.cat([b[:-1], b[1:]], 1)
    ae = torch.cat([a[:-1], a[1:]], 1)
    l = torch.arange(at.lmax + 1, dtype=torch.float64, device='cuda')
    l2 = l * (l + 1)
    Kb = torch.einsum('abc,ec->eab', HGH, be) - GG
    Ka = torch.einsum('abc,ec->eab', HHH, ae)
    K = torch.zeros(at.lmax + 1, 2 * n, 2 * n, dtype=torch.float64, device='cuda')
    M = torch.zeros(2 * n, 2 * n, dtype=torch.float64, device='cuda')
    rows, cols = dof[:, :, None].expand(-1, 4, 4), dof[:, None, :].expand(-1, 4, 4)
    for k in range(at.lmax + 1):
        K[k].index_put_((rows, cols), Kb + l2[k] * Ka, accumulate=True)
    M.index_put_((rows, cols), HH.expand(n - 1, 4, 4), accumulate=True)
    for row in (0, 2 * n - 2):
        K[:, row] = 0.0
        K[:, row, row] = 1.0
    return K, M


def _coulomb(grid, rho):
    """Becke-Dickson potentials of the rows of rho at every grid point."""
    k, N = rho.shape
    v = torch.zeros(k, N, dtype=torch.float64, device='cuda')
    made, off = {}, 0
    for A, (at, R) in enumerate(zip(grid.atoms, grid.centers)):
        n, lmax, ls = at.n, at.lmax, (at.lmax + 1) ** 2
        key = (at.R, n, lmax)
        if key not in made:
            made[key] = _radial_matrices(at)
        K, M = made[key]
        here = slice(off, off + grid.size[A])
        off += grid.size[A]
        g = (rho[:, here] * grid.becke[here] * grid.w[here]).reshape(k * n, at.nang)
        lof = torch.tensor([l for l in range(lmax + 1) for _ in range(2 * l + 1)],
                           dtype=torch.float64, device='cuda')
        f = (g @ _harmonics(at.u, lmax)).reshape(k, n, ls)
        f = f * torch.sqrt(4 * math.pi * (2.0 * lof + 1)) / (at.w * at.wang.sum())[:, None]
        f = f.permute(1, 0, 2).reshape(n, k * ls)
        lk = lof.repeat(k)
        # right-hand sides: the source -4 pi f as Hermite data, the end values
        # from the radial moments
        j1, j2 = at.j1[:, None], at.j2[:, None]
        src = torch.stack([f * j1 * j1, (_spline(f) * j1 + 2 * f * j2) * j1], 1)
        rhs = M @ (-4 * math.pi * src.reshape(2 * n, k * ls))
        t = at.r[:, None]
        rhs[0] = (f * (t[0] / t) ** lk / t * at.w[:, None]).sum(0) / (2 * lk + 1)
        rhs[-2] = (f * (t / t[-1]) ** lk / t[-1] * at.w[:, None]).sum(0) / (2 * lk + 1)
        x = torch.empty_like(rhs)
        for l in range(lmax + 1):
            cols = (lk == l).nonzero()[:, 0]
            x[:, cols] = torch.linalg.solve(K[l], rhs[:, cols])
        y, d = x[0::2], x[1::2]
        zz = y[1:] - y[:-1]
        c = torch.stack([y[:-1], d[:-1], 3 * zz - 2 * d[:-1] - d[1:], d[:-1] + d[1:] - 2 * zz], 2)
        c = c.reshape(n - 1, k, ls, 4) * (torch.sqrt(2.0 * lof + 1) /
                                          math.sqrt(4 * math.pi))[:, None]
        ends = (y[[0, -1]].reshape(2, k, ls) * torch.sqrt(2.0 * lof + 1) /
                math.sqrt(4 * math.pi))
        step = max(1, (1 << 26) // (4 * ls))
        for i in range(0, N, step):
            X = grid.points[i:i + step] - R
            dist = X.norm(dim=1)
            S = _harmonics(X / dist[:, None], lmax)
            tt = n - 2 * torch.atan(torch.sqrt(at.R / dist)) / at.z
            j = tt.floor().long().clamp(0, n - 2)
            u = tt - j
            low, high = dist < at.r[0], dist > at.r[-1]
            left = (dist[:, None] / at.r[0]).clamp(max=1.0) ** lof
            right = (at.r[-1] / dist[:, None]).clamp(max=1.0) ** (lof + 1)
            for q in range(k):
                s = c[:, q][j]
                val = s[..., 0] + u[:, None] * (s[..., 1] + u[:, None] *
                                                (s[..., 2] + u[:, None] * s[..., 3]))
                val = torch.where(low[:, None], ends[0, q] * left, val)
                val = torch.where(high[:, None], ends[1, q] * right, val)
                v[q, i:i + step] += (val * S).sum(1)
    return v


def _density(phi, D):
    return torch.cat([((D @ phi[:, i:i + (1 << 18)]) * phi[:, i:i + (1 << 18)]).sum(0)
                      for i in range(0, phi.shape[1], 1 << 18)])


def _exact_build(m, D, precision):
    grid = _Grid(*m)
    phi = grid.phi()
    rho = _density(phi, D)
    v = _coulomb(grid, rho[None])[0]
    F = (phi * (grid.becke * grid.w * v)) @ phi.T
    # 'int8x4' leaves out (rho = v = 0) the points with |weight| max phi^2 < 1e-24;
    # many have Becke weights that are themselves rounding residues, so which
    # points these are has no value of its own
    return (F, rho, v) if precision == 'fp64' else (F, None, None)


def _exact_gradient(case, D, R):
    """(E, dE/dD, dE/dR) of the charge energy by automatic differentiation."""
    D = D.clone().requires_grad_(True)
    R = R.clone().requires_grad_(True)
    atoms, nrad, nang = _molecules(case)[0]
    grid = _Grid(atoms, nrad, nang, centers=R.cuda())
    Z = [ELEMENTS[s]['atomic_number'] for s in grid.symbols]
    v = sum(z / (grid.points - C).norm(dim=1) for z, C in zip(Z, grid.centers))
    E = -(grid.becke * grid.w * v * _density(grid.phi(), D)).sum()
    E.backward()
    return E.detach(), D.grad, R.grad


def exact(case, seed):
    op, precision = case['op'], case['precision']
    mols = _molecules(case)
    n = [sum(_functions(s) for s, _ in m[0]) for m in mols]
    occ = [max(1, _electrons(m[0]) // 2) for m in mols]
    if op == 'batch':
        return [_exact_build(m, _density_matrix(n[k], occ[k], seed, k), precision)[0]
                for k, m in enumerate(mols)]
    if op == 'build':
        return _exact_build(mols[0], _density_matrix(n[0], occ[0], seed), precision)
    if op == 'gradient':
        D = _density_matrix(n[0], occ[0], seed)
        return [_exact_gradient(case, D, _displaced(case, seed, k)) for k in (1, 2)]
    if op == 'move':
        grid = _Grid(*mols[0], centers=_displaced(case, seed, 1).cuda())
        return grid.becke, grid.phi()
    if precision == 'int8x4' and op in ('density', 'potential', 'potentials'):
        return None  # see _exact_build
    grid = _Grid(*mols[0])
    phi = grid.phi()
    if op == 'density':
        return _density(phi, _density_matrix(n[0], occ[0], seed))
    if op == 'quadrature':
        v = _potential(grid.points, grid.centers, seed)
        return (phi * (grid.becke * grid.w * v)) @ phi.T
    if op == 'potential':
        charges = [ELEMENTS[s]['atomic_number'] for s in grid.symbols]
        rho = _charge_density(grid.points, grid.centers, charges, seed)
        return _coulomb(grid, rho[None])[0]
    if op == 'potentials':
        return _coulomb(grid, _pair_densities(case, phi, seed))
    W = grid.becke * grid.w
    K = torch.zeros(n[0], n[0], dtype=torch.float64, device='cuda')
    for psi in _orbitals(case, seed).T @ phi:
        K += (phi * (W * psi)) @ _coulomb(grid, psi * phi).T
    return 0.5 * (K + K.T)
