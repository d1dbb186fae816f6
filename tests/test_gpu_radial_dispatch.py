"""Radial solves on both sides of the line between the tabulated operators (up
to 256 radial points) and substitution, alone, in batches of solves, mixed in
one molecule and in one batch of molecules."""
import numpy as np
import pytest

from helpers import H2O, HCN, oracle_system, product_system, random_density

pytestmark = pytest.mark.gpu


def _densities(og, k):
    rng = np.random.default_rng(17)
    r = np.linalg.norm(og.points, axis=1)
    return np.stack([np.exp(-r) * (1.0 + rng.normal(size=len(r))) for _ in range(k)])


@pytest.mark.parametrize('nrad', [256, 257, [300, 257, 40], [40, 256, 300]])
def test_potentials_around_the_line(oracle, basis_library, elements, nrad):
    import torch
    import napmo_b200 as nb
    nang, lmax = 26, 3
    ms, grid = product_system(H2O, nrad=nrad, nang=nang)
    og, _ = oracle_system(oracle, basis_library, elements, H2O, nrad=nrad, nang=nang)
    rho = _densities(og, 3)
    fb = nb.FockBuilder(grid, ms['e-']['basis'], lmax)
    x = torch.as_tensor(rho).cuda()
    many = fb.coulomb_potentials(x).cpu().numpy()
    # both sides' rounding grows with the square of the radial points; 1e-11 of
    # the largest potential at 40 of them (test_gpu_poisson_edges.py)
    tol = 1e-11 * (np.max(nrad) / 40.0) ** 2
    for k, r in enumerate(rho):
        ref = oracle.compute_coulomb(og, r, lmax)
        assert np.abs(many[k] - ref).max() <= tol * np.abs(ref).max()
        assert np.array_equal(fb.coulomb_potential(x[k]).cpu().numpy(), many[k])


@pytest.mark.parametrize('mode', ['streams', 'stages'])
def test_batch_with_long_radial_grids(mode):
    """Each molecule's own build, whatever grids the others have."""
    import torch
    import napmo_b200 as nb
    plans = []
    for atoms, nrad in ((H2O, 40), (HCN, [257, 50, 50]), (H2O, 300), (HCN, 256)):
        ms, grid = product_system(atoms, nrad=nrad, nang=26)
        plans.append(nb.FockBuilder(grid, ms['e-']['basis'], 3))
    Ds = [torch.as_tensor(random_density(p.n, 5, 60 + k)).cuda() for k, p in enumerate(plans)]
    own = [p.build(D)[0] for p, D in zip(plans, Ds)]
    batch = nb.FockBatch(plans)
    batch.set_mode(mode)
    for F, R in zip(batch.build(Ds), own):
        assert torch.equal(F, R)
