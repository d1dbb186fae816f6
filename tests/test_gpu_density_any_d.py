"""Density of matrices that need not be symmetric (transition densities,
entry-wise differences): every entry point gives sum_ij D_ij phi_i phi_j, at
the edges of the FP64 kernels' size classes, in both batch modes and as the
tensor-core path does, against 64-bit torch."""
import numpy as np
import pytest

from helpers import H2O, product_system

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def _reference(D, x):
    """rho and the bound of both sides' rounding: 2 n + 4 units of sum |terms| each."""
    ref = ((D @ x) * x).sum(0)
    size = ((D.abs() @ x.abs()) * x.abs()).sum(0)
    return ref, 2 * (2 * D.shape[0] + 4) * EPS * size


def _matrix(n, seed):
    import torch
    g = torch.Generator().manual_seed(seed)
    return torch.randn(n, n, dtype=torch.float64, generator=g).cuda()


@pytest.mark.parametrize('n', [1, 16, 17, 32, 33, 49, 64, 65, 112, 127, 128, 129, 144, 145, 210,
                               257])
def test_density_of_any_matrix(n):
    import torch
    from napmo_b200 import cext
    npoint, ld = 2049, 2176
    g = torch.Generator().manual_seed(n)
    phi = torch.zeros(n, ld, dtype=torch.float64)
    phi[:, :npoint] = torch.randn(n, npoint, dtype=torch.float64, generator=g)
    phi = phi.cuda()
    D = _matrix(n, 500 + n)
    shifted = torch.empty(n * n + 1, dtype=torch.float64, device='cuda')[1:]
    shifted.copy_(D.reshape(-1))  # 8-byte aligned rows
    upper = torch.triu(D)
    for d in (D, shifted.view(n, n), upper, upper.T.contiguous()):
        rho = torch.full((npoint,), float('nan'), dtype=torch.float64, device='cuda')
        cext.checked(cext.lib.napmo_gpu_density(n, npoint, phi.data_ptr(), ld, d.data_ptr(),
                                                rho.data_ptr(),
                                                torch.cuda.current_stream().cuda_stream))
        ref, tol = _reference(d, phi[:, :npoint])
        assert bool(((rho - ref).abs() <= tol).all())


def _systems():
    from napmo_b200.system import alkane_geometry
    return [product_system(a, nrad=12, nang=26)
            for a in (H2O, alkane_geometry(3), alkane_geometry(5))]  # 25, 85, 135 functions


def test_plans_and_host_entry():
    import torch
    import napmo_b200 as nb
    from napmo_b200 import cext
    for k, (ms, grid) in enumerate(_systems()):
        fb = nb.FockBuilder(grid, ms['e-']['basis'], 5)
        D = _matrix(fb.n, k)
        ref, tol = _reference(D, fb.phi()[:, :fb.npoint])
        assert bool(((fb.density(D) - ref).abs() <= tol).all())
        host = np.empty(fb.npoint)
        cext.lib.nwavefunction_compute_density_from_dm(
            ms['e-']['basis']._this, grid._this, np.ascontiguousarray(D.cpu().numpy()), host, 0.0,
            np.zeros(fb.n))
        cext.check()
        assert bool(((torch.as_tensor(host).cuda() - ref).abs() <= tol).all())


@pytest.mark.parametrize('mode', ['streams', 'stages'])
def test_batches(mode):
    import torch
    import napmo_b200 as nb
    systems = _systems()
    fbs = [nb.FockBuilder(grid, ms['e-']['basis'], 5) for ms, grid in systems]
    Ds = [_matrix(fb.n, 10 + k) for k, fb in enumerate(fbs)]
    own = []
    for fb, D in zip(fbs, Ds):
        F, rho, _ = fb.build(D)
        ref, tol = _reference(D, fb.phi()[:, :fb.npoint])
        assert bool(((rho - ref).abs() <= tol).all())
        own.append(F)
    batch = nb.FockBatch(fbs)
    batch.set_mode(mode)
    for F, R in zip(batch.build(Ds), own):
        assert torch.equal(F, R)


def test_captured_density_follows_its_input():
    """The folded matrix of a captured call is formed anew by every replay."""
    import torch
    from napmo_b200 import cext
    n, npoint, ld = 145, 900, 1024
    phi = torch.zeros(n, ld, dtype=torch.float64, device='cuda')
    phi[:, :npoint] = torch.randn(n, npoint, dtype=torch.float64, device='cuda')
    D = _matrix(n, 1)
    rho = torch.zeros(npoint, dtype=torch.float64, device='cuda')
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        cext.checked(cext.lib.napmo_gpu_density(n, npoint, phi.data_ptr(), ld, D.data_ptr(),
                                                rho.data_ptr(),
                                                torch.cuda.current_stream().cuda_stream))
    for seed in (2, 3):
        D.copy_(_matrix(n, seed))
        graph.replay()
        ref, tol = _reference(D, phi[:, :npoint])
        assert bool(((rho - ref).abs() <= tol).all())


def test_calls_on_two_streams_keep_their_own_folded_matrix():
    import torch
    from napmo_b200 import cext
    n, npoint, ld = 145, 40000, 40064
    phi = torch.zeros(n, ld, dtype=torch.float64, device='cuda')
    phi[:, :npoint] = torch.randn(n, npoint, dtype=torch.float64, device='cuda')
    streams = [torch.cuda.Stream() for _ in range(2)]
    Ds = [_matrix(n, 20 + k) for k in range(16)]
    rhos = [torch.empty(npoint, dtype=torch.float64, device='cuda') for _ in Ds]
    torch.cuda.synchronize()
    for k, (D, rho) in enumerate(zip(Ds, rhos)):
        cext.checked(cext.lib.napmo_gpu_density(n, npoint, phi.data_ptr(), ld, D.data_ptr(),
                                                rho.data_ptr(), streams[k % 2].cuda_stream))
    torch.cuda.synchronize()
    for D, rho in zip(Ds, rhos):
        ref, tol = _reference(D, phi[:, :npoint])
        assert bool(((rho - ref).abs() <= tol).all())


def test_scratch_is_given_back_with_the_last_plan():
    import gc
    import torch
    import napmo_b200 as nb
    ms, grid = _systems()[2]
    fb = nb.FockBuilder(grid, ms['e-']['basis'], 5)
    for _ in range(3):  # each synchronisation may return memory; the results stay right
        D = _matrix(fb.n, 7)
        ref, tol = _reference(D, fb.phi()[:, :fb.npoint])
        assert bool(((fb.density(D) - ref).abs() <= tol).all())
    del fb
    gc.collect()
    again = nb.FockBuilder(grid, ms['e-']['basis'], 5)
    assert bool(((again.density(D) - ref).abs() <= tol).all())
