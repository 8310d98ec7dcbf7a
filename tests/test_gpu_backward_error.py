"""Backward error of the factorizations where a panel solve by inverted diagonal
blocks, or sums taken out of order, would lose it.  Bar: the oracle's own error
on the same matrices (the reference's order of operations, one rounding after
another); the residuals are formed in extended precision."""
import numpy as np
import pytest

from conftest import seeded, to_dev, to_host

pytestmark = pytest.mark.gpu

N = 384


def _chol_error(A, L):
    L = np.tril(L).astype(np.longdouble)
    return float(np.linalg.norm((L @ L.T - A).astype(float)) / np.linalg.norm(A))


def _lu_error(A, LU, p):
    P = A.copy()
    for i, r in enumerate(p):
        P[[i, i + r]] = P[[i + r, i]]
    X = LU.astype(np.longdouble)
    R = (np.tril(X, -1) + np.eye(len(A))) @ np.triu(X) - P
    return float(np.linalg.norm(R.astype(float)) / np.linalg.norm(A))


def _lu(cuda, flame, A):
    Ad = to_dev(cuda, A)
    p = cuda.zeros(len(A), dtype=cuda.int32, device="cuda")
    flame.lu_piv(Ad, p)
    return to_host(Ad), p.cpu().numpy()


@pytest.mark.parametrize("nugget", [1e-6, 1e-9, 1e-11])
def test_chol_smooth_kernel(cuda, flame, oracle, nugget):
    """Squared-exponential kernel of points in a row: nearly dependent neighbours."""
    x = np.linspace(0, 1, N)
    A = np.exp(-0.5 * ((x[:, None] - x[None]) / 0.3) ** 2) + nugget * np.eye(N)
    Lo, ro = oracle.chol(A)
    Ad = to_dev(cuda, A)
    assert flame.chol(Ad) == ro == flame.FLA_SUCCESS
    assert _chol_error(A, to_host(Ad)) <= _chol_error(A, Lo)


def _near_minus_one(rng):
    """A factor L whose 32 x 32 diagonal blocks have entries near -1 below the
    diagonal: their inverses grow like 2^32."""
    L = np.eye(N)
    for k in range(0, N, 32):
        L[k:k + 32, k:k + 32] += np.tril(-1 + 1e-3 * rng.uniform(0, 1, (32, 32)), -1)
    return L @ (np.triu(rng.uniform(-1, 1, (N, N)), 1) + 2 * np.eye(N))


def _chebyshev(rng):
    x = np.sort(rng.uniform(-1, 1, N))
    return np.cos(np.arange(N)[None] * np.arccos(x[:, None]))


FAMILIES = {"near_minus_one": _near_minus_one, "uniform": lambda rng: rng.uniform(-1, 1, (N, N)), "chebyshev": _chebyshev}


@pytest.mark.parametrize("family", sorted(FAMILIES))
def test_lu(cuda, flame, oracle, family):
    here, ref = [], []
    for s in range(4):
        A = FAMILIES[family](seeded(s))
        LUo, po, ro = oracle.lu_piv(A)
        LU, p = _lu(cuda, flame, A)  # its own pivots: a smooth matrix's last ones are rounding
        here.append(_lu_error(A, LU, p))
        ref.append(_lu_error(A, LUo, po))
    assert np.mean(here) <= np.mean(ref), (here, ref)


@pytest.mark.parametrize("k", [0, 5, 38, 127])
def test_infinite_entry(cuda, flame, oracle, k):
    """An infinite entry right of (below) the first block column: the entries of
    its column (row) before it stay what they are without it."""
    A = seeded(k).uniform(-1, 1, (200, 200))
    A[np.arange(200), np.arange(200)] += 20.0  # no interchanges
    A[k, 150] = np.inf
    LUo, po, _ = oracle.lu_piv(A)
    LU, p = _lu(cuda, flame, A)
    assert np.array_equal(p[:128], po[:128])
    assert np.isfinite(LU[:k, 150]).all() and np.isfinite(LUo[:k, 150]).all()
    assert np.allclose(LU[:k, 150], LUo[:k, 150], rtol=0, atol=1e-13)
    S = A + A.T
    S[150, k] = S[k, 150] = np.inf
    Lo, ro = oracle.chol(S)
    Sd = to_dev(cuda, S)
    assert flame.chol(Sd) == ro
    L = to_host(Sd)
    assert np.isfinite(L[150, :k]).all() and np.allclose(L[150, :k], Lo[150, :k], rtol=0, atol=1e-13)

