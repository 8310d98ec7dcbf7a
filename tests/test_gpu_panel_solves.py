"""The panels' triangular solves (X := X inv(L)^T) at the edges of their
16-column steps and of their 16, 32 and 64 rows per CTA: U12 of wide LU
factorizations and the block columns of Cholesky factorizations.

Bound, entry by entry: a factorization computed with b products per entry in
any order leaves |A - L U| <= (b + 2) eps |L| |U|, and as much again for the
residual formed here."""
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -52


def _colmajor(A):
    return A.new_empty_strided(tuple(A.shape), (1, A.shape[0])).copy_(A)


@pytest.mark.parametrize("b", [1, 2, 7, 8, 15, 16, 17, 31, 33, 48, 63, 64, 65, 100, 127, 128, 129])
@pytest.mark.parametrize("cols", [1, 15, 17, 300, 2500, 4800])
def test_wide_lu(cuda, flame, b, cols):
    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(b * 7 + cols)
    A = torch.rand((b, b + cols), dtype=torch.float64, device="cuda", generator=g) * 2 - 1
    X, p = _colmajor(A), torch.zeros(b, dtype=torch.int32, device="cuda")
    assert flame.lu_piv(X, p) == flame.FLA_SUCCESS, flame.last_error()
    perm = list(range(b))
    for i, r in enumerate(p.tolist()):
        perm[i], perm[i + r] = perm[i + r], perm[i]
    L = torch.tril(X[:, :b], -1) + torch.eye(b, dtype=torch.float64, device="cuda")
    U = torch.triu(X)
    assert bool(((L @ U - A[perm]).abs() <= 2 * (b + 2) * EPS * (L.abs() @ U.abs())).all())


@pytest.mark.parametrize("n", [129, 144, 145, 257, 2496, 2497, 4865, 5000])
@pytest.mark.parametrize("upper", [0, 1])
def test_chol_block_columns(cuda, flame, n, upper):
    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(n)
    G = torch.randn((n, n), dtype=torch.float64, device="cuda", generator=g)
    A = G @ G.t() / n + torch.eye(n, dtype=torch.float64, device="cuda")
    X = _colmajor(A)
    assert flame.chol(X, flame.FLA_UPPER_TRIANGULAR if upper else flame.FLA_LOWER_TRIANGULAR) == flame.FLA_SUCCESS
    L = torch.triu(X).t() if upper else torch.tril(X)
    R = torch.tril(L @ L.t() - A).abs()
    # the first 128 columns: one block column under the diagonal block
    w = 128
    assert bool((R[:, :w] <= 2 * (w + 2) * EPS * (L[:, :w].abs() @ L[:w, :w].abs().t())).all())
    assert bool((R <= 2 * (n + 2) * EPS * (L.abs() @ L.abs().t())).all())
