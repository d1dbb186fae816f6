"""FP64 density and quadrature over long point ranges (every slot of the copy
ring reused many times, several groups and chunks per CTA) and over the lists
of screened plans, at every size class, against 64-bit torch."""
import pytest

from helpers import H2O, product_system, random_density

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def _sums(phi, b, w):
    """phi diag(w) b^T, upper triangle mirrored, and its rounding bound: at most
    (points + 2) units of sum |terms| on either side."""
    import torch
    ref, size = (phi * w) @ b.T, (phi * w).abs() @ b.abs().T
    up = lambda x: torch.triu(x) + torch.triu(x, 1).T
    return up(ref), 2 * (phi.shape[1] + 2) * EPS * up(size)


def _density(phi, D):
    ref, size = ((D @ phi) * phi).sum(0), ((D.abs() @ phi.abs()) * phi.abs()).sum(0)
    return ref, 2 * (2 * D.shape[0] + 4) * EPS * size


@pytest.mark.parametrize('n', [16, 25, 49, 64, 65, 127, 128, 129, 210, 300])
def test_long_ranges(n):
    import torch
    from napmo_b200 import cext
    npoint, ld = 60001, 60032
    g = torch.Generator().manual_seed(n)
    x = torch.randn(2, n, npoint, dtype=torch.float64, generator=g)
    phi, psi = torch.zeros(2, n, ld, dtype=torch.float64, device='cuda')
    phi[:, :npoint], psi[:, :npoint] = x.cuda()
    wv = torch.zeros(ld, dtype=torch.float64, device='cuda')
    wv[:npoint] = torch.randn(npoint, dtype=torch.float64, generator=g).cuda()
    s = torch.cuda.current_stream().cuda_stream
    for b in (phi, psi):
        ref, tol = _sums(phi[:, :npoint], b[:, :npoint], wv[:npoint])
        for entry in ('napmo_gpu_quadrature', 'napmo_gpu_quadrature_noalloc'):
            F = torch.full((n, n), float('nan'), dtype=torch.float64, device='cuda')
            cext.checked(getattr(cext.lib, entry)(
                n, npoint, phi.data_ptr(), None if b is phi else b.data_ptr(), ld, wv.data_ptr(),
                F.data_ptr(), s))
            assert torch.equal(F, F.T)
            assert bool(((F - ref).abs() <= tol).all()), entry
    D = torch.randn(n, n, dtype=torch.float64, generator=g).cuda()
    rho = torch.full((npoint,), float('nan'), dtype=torch.float64, device='cuda')
    cext.checked(cext.lib.napmo_gpu_density(n, npoint, phi.data_ptr(), ld, D.data_ptr(),
                                            rho.data_ptr(), s))
    ref, tol = _density(phi[:, :npoint], D)
    assert bool(((rho - ref).abs() <= tol).all())


def _screened(carbons, tol):
    import napmo_b200 as nb
    from napmo_b200.system import alkane_geometry
    ms, grid = product_system(alkane_geometry(carbons) if carbons else H2O, nrad=30, nang=110)
    fb = nb.FockBuilder(grid, ms['e-']['basis'], 8)
    fb.set_fp64_screening(tol)
    return fb


@pytest.mark.parametrize('carbons', [0, 1, 2, 3, 5])  # 25, 35, 60, 85, 135 functions
@pytest.mark.parametrize('tol', [1e-20, 1e-6])
def test_screened_lists(carbons, tol):
    import torch
    fb = _screened(carbons, tol)
    N, keep = fb.npoint, fb.kept_points()
    assert 0 < int(keep.sum()) < N
    phi = fb.phi()[:, :N]
    g = torch.Generator().manual_seed(carbons)
    D = torch.randn(fb.n, fb.n, dtype=torch.float64, generator=g).cuda()
    ref, bound = _density(phi, D)
    rho = fb.density(D)
    assert bool(((rho - ref).abs() <= bound)[keep].all()) and not bool(rho[~keep].any())
    # the quadrature runs over the 16-point blocks that hold a kept point
    pad = torch.zeros((N + 15) // 16 * 16, dtype=torch.bool, device='cuda')
    pad[:N] = keep
    listed = pad.view(-1, 16).any(dim=1).repeat_interleave(16)[:N]
    v = torch.randn(N, dtype=torch.float64, generator=g).cuda()
    one = torch.as_tensor(fb.grid.becke_weights * fb.grid.weights).cuda()
    # forming the weights rounds twice more on either side
    ref, bound = _sums(phi[:, listed], phi[:, listed], (one * v)[listed])
    assert bool(((fb.quadrature(1.0, v) - ref).abs() <= 2 * bound).all())


@pytest.mark.parametrize('mode', ['streams', 'stages'])
def test_screened_batches(mode):
    import torch
    import napmo_b200 as nb
    plans = [_screened(c, t) for c, t in ((2, 1e-8), (0, 1e-3), (5, 1e-12), (3, 1e-6))]
    Ds = [torch.as_tensor(random_density(p.n, 5, 80 + k)).cuda() for k, p in enumerate(plans)]
    own = [p.build(D)[0] for p, D in zip(plans, Ds)]
    batch = nb.FockBatch(plans)
    batch.set_mode(mode)
    for F, R in zip(batch.build(Ds), own):
        assert torch.equal(F, R)
