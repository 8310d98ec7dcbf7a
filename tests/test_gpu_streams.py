"""Work that overlaps on several streams gives what it gives alone."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def test_adjoint_batched_large_orders(cuda, flame):
    """Orders above 2048 over the pool of streams, each in its own scratch,
    against one matrix at a time.  Both split their products over k, in other
    numbers of slices: the bar of the adjoint's other comparisons, 1e-10."""
    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(3)
    Ls, Lbars, alone = [], [], []
    for n in (2305, 2176, 2050, 2305, 1000, 2100, 129, 2200, 2064):
        G = torch.randn((n, n), dtype=torch.float64, device="cuda", generator=g)
        L = torch.linalg.cholesky(G @ G.t() / n + torch.eye(n, dtype=torch.float64, device="cuda"))
        Ls.append(L.t().contiguous().clone().t())
        Lb = torch.tril(torch.randn((n, n), dtype=torch.float64, device="cuda", generator=g))
        Lbars.append(Lb.t().contiguous().clone().t())
        one = Lb.t().contiguous().clone().t()
        assert flame.chol_adjoint(Ls[-1], one) == flame.FLA_SUCCESS, flame.last_error()
        alone.append(one)
    assert flame.chol_adjoint_batched(Ls, Lbars, 0.0) == flame.FLA_SUCCESS, flame.last_error()
    for a, b in zip(Lbars, alone):
        assert ((torch.tril(a) - torch.tril(b)).norm() / torch.tril(b).norm()).item() < 1e-10


@pytest.mark.parametrize("m,n,k", [(512, 512, 1024), (640, 384, 256)])
def test_small_gemm_tiles_beside_panels(cuda, flame, m, n, k):
    """The 32 x 32 tiles (at most 111 tiles of 64 x 64; their boxes are refilled
    past k = 128) beside Cholesky panel work: bitwise what they give alone."""
    bad = C.c_ulonglong(1)
    assert flame.lib().FLA_B200_gemm_concurrency_check(m, n, k, 2000, C.byref(bad)) == flame.FLA_SUCCESS, flame.last_error()
    assert bad.value == 0
