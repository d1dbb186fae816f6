"""One rule for the evaluation's item lists: solves that truncate evaluate by
interval, others take an atom's own points on their nodes, whatever the plan's
screening, its batch and what it ran before.  Bits are compared throughout."""
import numpy as np
import pytest

from helpers import H2O, HCN, product_system, random_density

pytestmark = pytest.mark.gpu

TOL = 1e-5


def _plan(atoms=H2O, nrad=30, nang=110, lmax=8):
    import torch
    import napmo_b200 as nb
    ms, grid = product_system(atoms, nrad=nrad, nang=nang)
    fb = nb.FockBuilder(grid, ms['e-']['basis'], lmax)
    g = torch.Generator().manual_seed(3)
    r = torch.as_tensor(np.linalg.norm(grid.points, axis=1))
    rho = torch.exp(-r) * (1.0 + torch.randn(fb.npoint, dtype=torch.float64, generator=g))
    return fb, rho.cuda()


@pytest.mark.parametrize('tol', [0.0, TOL])
@pytest.mark.parametrize('nrad,nang,lmax', [(2, 6, 1), (3, 26, 2), (30, 110, 8)])
def test_screened_points_equal_the_unscreened_solve(nrad, nang, lmax, tol):
    import torch
    fb, rho = _plan(nrad=nrad, nang=nang, lmax=lmax)
    fb.set_poisson_tolerance(tol)
    full = fb.coulomb_potential(rho)
    fb.set_fp64_screening(1e-8)
    keep = fb.kept_points()
    assert int(keep.sum()) < fb.npoint or nrad == 2
    assert torch.equal(fb.coulomb_potential(rho)[keep], full[keep])
    both = torch.stack([rho, 2.0 * rho])
    assert torch.equal(fb.coulomb_potentials(both)[0][keep], full[keep])


@pytest.mark.parametrize('mode', ['streams', 'stages'])
@pytest.mark.parametrize('tol', [0.0, TOL])
def test_batch_of_screened_and_unscreened_plans(mode, tol):
    import torch
    import napmo_b200 as nb
    plans = [_plan(H2O)[0], _plan(HCN)[0], _plan(H2O, nrad=23, nang=50, lmax=5)[0]]
    plans[1].set_fp64_screening(1e-14)
    for p in plans:
        p.set_poisson_tolerance(tol)
    Ds = [torch.as_tensor(random_density(p.n, 5, 40 + k)).cuda() for k, p in enumerate(plans)]
    own = [p.build(D)[0] for p, D in zip(plans, Ds)]
    batch = nb.FockBatch(plans)
    batch.set_mode(mode)
    for F, R in zip(batch.build(Ds), own):
        assert torch.equal(F, R)


@pytest.mark.parametrize('screen', [0.0, 1e-14])
@pytest.mark.parametrize('tols', [(0.0, TOL), (TOL, 0.0)])
def test_captured_solve_equals_the_eager_one(screen, tols):
    """Only the first tolerance's solve has run when the second is captured."""
    import torch
    fb, rho = _plan()
    if screen:
        fb.set_fp64_screening(screen)
    fb.set_poisson_tolerance(tols[0])
    fb.coulomb_potential(rho)
    fb.set_poisson_tolerance(tols[1])
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        v = fb.coulomb_potential(rho)
    graph.replay()
    torch.cuda.synchronize()
    captured = v.clone()
    assert torch.equal(captured, fb.coulomb_potential(rho))
