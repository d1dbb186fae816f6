"""Solves in flight on one stream while another rebuilds what they read: a
screening mask's pair lists, another mask's lists in the same buffers, and a
move of the grid."""
import numpy as np
import pytest

from helpers import product_system

pytestmark = pytest.mark.gpu


def _setup():
    import torch
    import napmo_b200 as nb
    from napmo_b200.system import alkane_geometry
    ms, grid = product_system(alkane_geometry(3), nrad=40, nang=110)
    fb = nb.FockBuilder(grid, ms['e-']['basis'], 8)
    g = torch.Generator().manual_seed(1)
    rho = torch.rand(120, fb.npoint, dtype=torch.float64, generator=g).cuda()
    return ms, grid, fb, rho


def _in_flight(fb, rho, action):
    """Potentials of a batch of solves, with `action` run from the host while
    they are in flight on a stream of their own."""
    import torch
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        v = fb.coulomb_potentials(rho, stream=s)
    action()
    torch.cuda.synchronize()
    return v


def test_screened_lists_wait_for_solves_in_flight():
    import torch
    import napmo_b200 as nb
    ms, grid, fb, rho = _setup()
    quiet = fb.coulomb_potentials(rho)
    masks = [nb.FockBuilder(grid, ms['e-']['basis'], 8) for _ in range(2)]
    for m, tol in zip(masks, (1e-24, 1e-6)):
        m.set_fp64_screening(tol)
    keep = []

    def first_lists():
        keep.append(masks[0].coulomb_potential(rho[0]))

    def other_mask():
        keep.append(masks[1].coulomb_potential(rho[0]))

    assert torch.equal(_in_flight(fb, rho, first_lists), quiet)
    screened = masks[0].coulomb_potentials(rho)
    assert torch.equal(screened[0], keep[0])
    # the second mask's lists take the place of the first one's, in use here
    assert torch.equal(_in_flight(masks[0], rho, other_mask), screened)
    assert torch.equal(masks[1].coulomb_potential(rho[0]), keep[1])


def test_moves_wait_for_solves_in_flight():
    import torch
    ms, grid, fb, rho = _setup()
    quiet = fb.coulomb_potentials(rho)
    R = np.array([p['origin'] for p in ms['e-']['particles']], dtype=np.float64)
    assert torch.equal(_in_flight(fb, rho, lambda: grid.set_centers(R * 1.1)), quiet)
    moved = fb.coulomb_potential(rho[0])
    assert not torch.equal(moved, quiet[0])
    grid.set_centers(R)
    assert torch.equal(fb.coulomb_potentials(rho), quiet)
