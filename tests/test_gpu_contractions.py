"""FP64 density and quadrature kernels at the edges of their size classes
(16-row fragments, the small-molecule kernels up to 64 functions, ragged and
full 128-wide tiles, short and long point ranges) against 64-bit torch."""
import pytest

pytestmark = pytest.mark.gpu

SIZES = (1, 15, 16, 17, 32, 33, 48, 49, 64, 65, 80, 112, 113, 127, 128, 129, 144, 210, 257, 300)
POINTS = (1, 130, 2049)
EPS = 2.0 ** -53


def _operands(n, npoint, seed):
    import torch
    g = torch.Generator().manual_seed(seed)
    ld = (npoint + 127) // 128 * 128
    phi = torch.zeros(n, ld, dtype=torch.float64)
    psi = torch.zeros(n, ld, dtype=torch.float64)
    wv = torch.zeros(ld, dtype=torch.float64)
    phi[:, :npoint] = torch.randn(n, npoint, dtype=torch.float64, generator=g)
    psi[:, :npoint] = torch.randn(n, npoint, dtype=torch.float64, generator=g)
    wv[:npoint] = torch.randn(npoint, dtype=torch.float64, generator=g)
    D = torch.randn(n, n, dtype=torch.float64, generator=g)
    return phi.cuda(), psi.cuda(), wv.cuda(), (D + D.T).cuda(), ld


@pytest.mark.parametrize('n', SIZES)
def test_quadrature_sizes(n):
    import torch
    from napmo_b200 import cext
    for npoint in POINTS:
        phi, psi, wv, _, ld = _operands(n, npoint, n)
        s = torch.cuda.current_stream().cuda_stream
        for second in (None, psi):
            b = phi if second is None else second
            ref = (phi * wv) @ b.T
            ref = torch.triu(ref) + torch.triu(ref, 1).T
            # rounding of both sums: at most (npoint + 2) units of sum |terms| each
            size = (phi * wv).abs() @ b.abs().T
            tol = 2 * (npoint + 2) * EPS * (torch.triu(size) + torch.triu(size, 1).T)
            for entry in ('napmo_gpu_quadrature', 'napmo_gpu_quadrature_noalloc'):
                F = torch.full((n, n), float('nan'), dtype=torch.float64, device='cuda')
                cext.checked(getattr(cext.lib, entry)(
                    n, npoint, phi.data_ptr(), None if second is None else second.data_ptr(), ld,
                    wv.data_ptr(), F.data_ptr(), s))
                assert torch.equal(F, F.T)
                assert bool(((F - ref).abs() <= tol).all()), (n, npoint, entry)


@pytest.mark.parametrize('n', SIZES)
def test_density_sizes(n):
    import torch
    from napmo_b200 import cext
    for npoint in POINTS:
        phi, _, _, D, ld = _operands(n, npoint, 1000 + n)
        rho = torch.full((npoint,), float('nan'), dtype=torch.float64, device='cuda')
        cext.checked(cext.lib.napmo_gpu_density(n, npoint, phi.data_ptr(), ld, D.data_ptr(),
                                                rho.data_ptr(),
                                                torch.cuda.current_stream().cuda_stream))
        x = phi[:, :npoint]
        ref = ((D @ x) * x).sum(0)
        size = ((D.abs() @ x.abs()) * x.abs()).sum(0)
        assert bool(((rho - ref).abs() <= 2 * (2 * n + 4) * EPS * size).all()), (n, npoint)
