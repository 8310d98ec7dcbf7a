"""FLA_Chol_batched at the edges of its 32-column panels, update tiles, the 256 /
512-thread split and the order (512) above which the older kernel takes over,
with padded leading dimensions and up to eight right-hand sides, and a matrix
that fails; each against the oracle's FLA_Chol.

Bars as in the other batched tests: factors within 1e-12 normwise, solutions
within 1e-11 of the oracle's, identical failure columns, the strictly upper
triangles and the right-hand sides of a failing matrix left alone."""
import numpy as np
import pytest

from conftest import rel_fro, seeded, spd, to_host

pytestmark = pytest.mark.gpu

SIZES = [1, 31, 32, 33, 48, 63, 64, 65, 97, 248, 255, 256, 257, 289, 481, 511, 512, 513, 600]


@pytest.mark.parametrize("nrhs,pad", [(0, 0), (1, 1), (8, 3)])
def test_panels_and_tiles(cuda, flame, oracle, nrhs, pad):
    torch = cuda
    rng = seeded(171 + nrhs)
    mats = [spd(rng, n) for n in SIZES]
    bad = SIZES.index(97)
    mats[bad][50, 50] = -1.0
    dev = []
    for A in mats:
        n = A.shape[0]
        buf = torch.full((n, n + pad), 7.0, dtype=torch.float64, device="cuda")  # rows: columns of A
        buf[:, :n] = torch.from_numpy((np.tril(A) + np.triu(np.full_like(A, np.nan), 1)).T.copy())
        dev.append(buf.t()[:n, :])
    rhs = [rng.standard_normal((n, nrhs)) for n in SIZES] if nrhs else None
    drhs = [torch.empty_strided((n, nrhs), (1, n + pad), dtype=torch.float64, device="cuda").copy_(torch.from_numpy(b))
            for n, b in zip(SIZES, rhs)] if nrhs else None
    r, info = flame.batched("chol", dev, rhs=drhs)
    assert r == flame.FLA_SUCCESS, flame.last_error()
    for i, A in enumerate(mats):
        n = SIZES[i]
        Lo, ro = oracle.chol(A)
        assert info[i] == ro, (n, info[i], ro)
        F = to_host(dev[i])
        assert np.isnan(F[np.triu_indices(n, 1)]).all(), n
        if ro != -1:
            assert nrhs == 0 or np.array_equal(to_host(drhs[i]), rhs[i])
            continue
        assert rel_fro(np.tril(F), np.tril(Lo)) < 1e-12, n
        if nrhs:
            assert rel_fro(to_host(drhs[i]), oracle.chol_solve(Lo, rhs[i])) < 1e-11, n


@pytest.mark.parametrize("n,nrhs", [(129, 1), (200, 40), (385, 200)])
@pytest.mark.parametrize("kind", ["chol", "lu"])
def test_mixed_solve_many_columns(cuda, flame, n, nrhs, kind):
    """The mixed-precision solvers' one-launch FP32 sweeps past 32 right-hand
    sides: refined to FP64 accuracy (backward error of a few eps)."""
    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(n + nrhs)
    G = torch.randn((n, n), dtype=torch.float64, device="cuda", generator=g)
    A = G @ G.t() / n + torch.eye(n, dtype=torch.float64, device="cuda") if kind == "chol" else G + n ** 0.5 * torch.eye(
        n, dtype=torch.float64, device="cuda")
    A = A.t().contiguous().clone().t()
    B = torch.empty_strided((n, nrhs), (1, n), dtype=torch.float64, device="cuda").normal_(generator=g)
    X = torch.empty_strided((n, nrhs), (1, n), dtype=torch.float64, device="cuda")
    f = flame.chol_solve_mixed if kind == "chol" else flame.lu_piv_solve_mixed
    r, it, _ = f(A, B, X)
    assert r == flame.FLA_SUCCESS and it >= 0, (r, it, flame.last_error())
    be = ((B - A @ X).abs().amax(0) / (A.abs().sum(1).max() * X.abs().amax(0) + B.abs().amax(0))).max().item()
    assert be < 8 * 2.2e-16, be
