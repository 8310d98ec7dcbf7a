"""The GEMM engine around the switch between its 32 x 32 and 64 x 64 tiles and
at the edges of the small tiles' k stages and splits, against FP64 torch.

Tolerance: both sides sum k products of N(0,1) values in some order, so an
entry differs by at most about 2 k eps sum |a b|; 4 k eps times the product
of the absolute values bounds it entry by entry."""
import pytest

pytestmark = pytest.mark.gpu


def colmajor(torch, m, n, g):
    return torch.randn((n, m), dtype=torch.float64, device="cuda", generator=g).t()


@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("m,n,k", [(2, 2, 2), (34, 30, 16), (32, 32, 32), (66, 34, 34), (64, 64, 128), (98, 130, 160),
                                   (130, 62, 130), (700, 600, 34), (710, 640, 34), (720, 700, 48), (126, 190, 4098)])
@pytest.mark.parametrize("lower", [0, 1])
def test_small_tiles(cuda, flame, ta, tb, m, n, k, lower):
    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(m * 7 + n * 3 + k)
    A = colmajor(torch, k, m, g) if ta else colmajor(torch, m, k, g)
    B = colmajor(torch, n, k, g) if tb else colmajor(torch, k, n, g)
    C = colmajor(torch, m, n, g)
    a, b = (A.t() if ta else A), (B.t() if tb else B)
    for alpha, beta in ((-1.0, 1.0), (0.5, 0.0)):
        out = C.t().clone().t()
        assert flame.lib().FLA_B200_dgemm(ta, tb, m, n, k, alpha, A.data_ptr(), A.stride(1), B.data_ptr(), B.stride(1),
                                          beta, out.data_ptr(), out.stride(1), lower) == flame.FLA_SUCCESS
        ref = alpha * (a @ b) + beta * C
        if lower:
            ref = torch.tril(ref) + torch.triu(C, 1)
        bound = 4 * (k + 2) * 2.2e-16 * (abs(alpha) * (a.abs() @ b.abs()) + abs(beta) * C.abs())
        assert bool(((out - ref).abs() <= bound).all()), ((out - ref).abs() / bound).max().item()
