"""The one-launch triangular solves (orders above 128, few right-hand sides) at
the edges of their 64-row blocks and 16-column groups, in all four directions,
and the composed row order of long pivot sequences.

Tolerance: a solve by blocks of order 64 is backward stable with a constant of
order 64, so |op(T) X - B| <= 8 64 eps (|op(T)| |X| + |B|) entry by entry, a
bound that does not depend on the condition of T."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SIZES = [(129, 1), (191, 16), (192, 17), (193, 3), (1000, 33), (1025, 64), (2500, 5)]


def colmajor(t):
    out = t.new_empty(t.numel()).as_strided(tuple(t.shape), (1, t.shape[0]))
    return out.copy_(t)


@pytest.mark.parametrize("n,nr", SIZES)
@pytest.mark.parametrize("upper", [0, 1])
def test_chol_solve_both_triangles(cuda, flame, n, nr, upper):
    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(n + nr)
    G = torch.randn((n, n), dtype=torch.float64, device="cuda", generator=g)
    A = G @ G.t() / n + torch.eye(n, dtype=torch.float64, device="cuda")
    L = torch.linalg.cholesky(A)
    F = colmajor(L.t() if upper else L)
    # the other triangle is not referenced
    F += torch.full_like(F, float("nan")).tril(-1) if upper else torch.full_like(F, float("nan")).triu(1)
    B = colmajor(torch.randn((n, nr), dtype=torch.float64, device="cuda", generator=g))
    X = colmajor(B)
    assert flame.chol_solve(F, B, X, flame.FLA_UPPER_TRIANGULAR if upper else flame.FLA_LOWER_TRIANGULAR) \
        == flame.FLA_SUCCESS, flame.last_error()
    # two triangular solves: the bound with |L| |L^T| for the product
    bound = 2 * 8 * 64 * 2.2e-16 * (L.abs() @ (L.t().abs() @ X.abs()) + B.abs())
    assert bool(((L @ (L.t() @ X) - B).abs() <= bound).all())


@pytest.mark.parametrize("n,nr", SIZES)
@pytest.mark.parametrize("trans", ["N", "T"])
def test_getrs_both_directions(cuda, flame, n, nr, trans):
    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(3 * n + nr)
    A = torch.rand((n, n), dtype=torch.float64, device="cuda", generator=g) * 2 - 1
    LU, piv = torch.linalg.lu_factor(A)
    LU, ip = colmajor(LU), piv.to(torch.int32).contiguous()
    B = colmajor(torch.randn((n, nr), dtype=torch.float64, device="cuda", generator=g))
    X = colmajor(B)
    info, ints = C.c_int(0), [C.c_int(v) for v in (n, nr, n, n)]
    lib = flame.lib()
    lib.dgetrs_(trans.encode(), C.byref(ints[0]), C.byref(ints[1]), C.c_void_p(LU.data_ptr()), C.byref(ints[2]),
                C.c_void_p(ip.data_ptr()), C.c_void_p(X.data_ptr()), C.byref(ints[3]), C.byref(info))
    assert info.value == 0
    P, L, U = torch.lu_unpack(LU, piv)
    if trans == "N":
        R, M = L @ (U @ X) - P.t() @ B, L.abs() @ (U.abs() @ X.abs()) + P.t() @ B.abs()
    else:
        R, M = U.t() @ (L.t() @ (P.t() @ X)) - B, U.t().abs() @ (L.t().abs() @ (P.t() @ X.abs())) + B.abs()
    assert bool((R.abs() <= 2 * 8 * 64 * 2.2e-16 * M).all())


@pytest.mark.parametrize("m,npiv,ncols", [(300, 129, 1), (1000, 1000, 3), (4096, 4095, 64), (60000, 6000, 2)])
@pytest.mark.parametrize("reverse", [0, 1])
def test_long_pivot_sequences(cuda, flame, m, npiv, ncols, reverse):
    torch = cuda
    rng = np.random.default_rng(m + npiv)
    p = np.array([rng.integers(0, m - i) if rng.random() < 0.7 else rng.integers(0, min(4, m - i))
                  for i in range(npiv)], dtype=np.int32)
    A = rng.integers(-1000, 1000, size=(m, ncols)).astype(np.float64)
    Ad, pd = colmajor(torch.from_numpy(A).cuda()), torch.from_numpy(p).cuda()
    assert flame.apply_pivots(pd, Ad, flame.FLA_TRANSPOSE if reverse else flame.FLA_NO_TRANSPOSE) == flame.FLA_SUCCESS
    for i in (range(npiv - 1, -1, -1) if reverse else range(npiv)):
        A[[i, i + p[i]]] = A[[i + p[i], i]]
    assert np.array_equal(Ad.cpu().numpy(), A)
