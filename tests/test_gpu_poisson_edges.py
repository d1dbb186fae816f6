"""Poisson stages at the edges of their range: the evaluation's column pairs
for every parity of lmax, one and two radial intervals per atom upwards, items
that end inside a thread's pairs, truncated solves and batches, on densities
with weight in every multipole, against the oracle."""
import numpy as np
import pytest

from helpers import H2O, oracle_system, product_system

pytestmark = pytest.mark.gpu


def _grids(oracle, basis_library, elements, nrad, nang):
    ms, grid = product_system(H2O, nrad=nrad, nang=nang)
    og, _ = oracle_system(oracle, basis_library, elements, H2O, nrad=nrad, nang=nang)
    return ms['e-']['basis'], grid, og


def _density(og, k=0):
    """Noise on every point (every multipole has weight), integrable."""
    rng = np.random.default_rng(7 + k)
    r = np.linalg.norm(og.points, axis=1)
    return np.exp(-r) * (1.0 + rng.normal(size=len(r)))


@pytest.mark.parametrize('lmax', [0, 1, 2, 3, 4, 5, 8, 11, 14, 19, 20])
@pytest.mark.parametrize('nrad,nang', [(5, 6), (23, 50), (40, 110)])
def test_potential_every_lmax(oracle, basis_library, elements, lmax, nrad, nang):
    import torch
    import napmo_b200 as nb
    basis, grid, og = _grids(oracle, basis_library, elements, nrad, nang)
    rho = np.stack([_density(og, k) for k in range(3)])
    ref = np.stack([oracle.compute_coulomb(og, r, lmax) for r in rho])
    fb = nb.FockBuilder(grid, basis, lmax)
    x = torch.as_tensor(rho).cuda()
    one = fb.coulomb_potential(x[0]).cpu().numpy()
    many = fb.coulomb_potentials(x).cpu().numpy()
    # both sides round the banded solves and sums of (lmax + 1)^2 terms: a few
    # 1e-13 of the largest potential
    assert np.abs(one - ref[0]).max() <= 1e-11 * np.abs(ref[0]).max()
    assert np.array_equal(one, many[0])
    for v, r in zip(many, ref):
        assert np.abs(v - r).max() <= 1e-11 * np.abs(r).max()


@pytest.mark.parametrize('lmax', [1, 6, 11, 20])
def test_truncated_potential(oracle, basis_library, elements, lmax):
    import torch
    import napmo_b200 as nb
    basis, grid, og = _grids(oracle, basis_library, elements, 23, 50)
    rho = torch.as_tensor(_density(og)).cuda()
    fb = nb.FockBuilder(grid, basis, lmax)
    full = fb.coulomb_potential(rho)
    for tol in (1e-12, 1e-6, 1e-2):
        fb.set_poisson_tolerance(tol)
        v = fb.coulomb_potential(rho)
        # each of the three atoms drops at most tol; rounding as above
        assert float((v - full).abs().max()) <= 3 * tol + 1e-12 * float(full.abs().max()), tol


@pytest.mark.parametrize('precision', ['fp64', 'int8x4'])
@pytest.mark.parametrize('nrad,nang', [(5, 6), (40, 110)])
def test_moved_plan_equals_a_new_one(oracle, basis_library, elements, precision, nrad, nang):
    import torch
    import napmo_b200 as nb
    lmax = nb.lebedev_get_order(nang) // 2
    basis, grid, og = _grids(oracle, basis_library, elements, nrad, nang)
    fb = nb.FockBuilder(grid, basis, lmax, precision=precision)
    rho = torch.as_tensor(np.stack([_density(og, k) for k in range(2)])).cuda()
    fb.coulomb_potentials(rho)
    R = np.array([xyz for _, xyz in H2O]) / 0.52917724924
    of = [int(np.argmin(((R - o) ** 2).sum(1))) for o in basis.origins()]
    # far apart (tail pairs grow), close together (they vanish), back
    for scale in (6.0, 0.8, 1.0):
        grid.set_centers(R * scale)
        basis.set_origins((R * scale)[of])
        fb.refresh()
        moved = fb.coulomb_potentials(rho)
        atoms = [(s, tuple(np.array(x) * scale)) for s, x in H2O]
        ms, fresh = product_system(atoms, nrad=nrad, nang=nang)
        fresh.set_centers(R * scale)  # the very same centres, to the last bit
        ms['e-']['basis'].set_origins((R * scale)[of])
        new = nb.FockBuilder(fresh, ms['e-']['basis'], lmax, precision=precision)
        assert torch.equal(moved, new.coulomb_potentials(rho)), scale
        assert torch.equal(fb.coulomb_potential(rho[0]), moved[0])
