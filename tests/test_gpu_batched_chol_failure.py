"""What FLA_Chol_batched leaves of a matrix that fails at column f: L in the
columns before f (in the failing 32-column panel, the rows of its diagonal
block), the failing pivot at (f, f), the strictly upper triangle and the
right-hand sides untouched.  Bar: 1e-12 normwise, as for the factors."""
import numpy as np
import pytest

from conftest import seeded, spd, to_host

pytestmark = pytest.mark.gpu

CASES = [(5, 0), (40, 33), (97, 50), (256, 39), (300, 299), (512, 480), (600, 555)]


def test_failing_matrices(cuda, flame):
    torch = cuda
    rng = seeded(77)
    mats, dev, rhs, drhs = [], [], [], []
    for n, f in CASES:
        A = spd(rng, n)
        # the pivot of column f becomes -0.75
        L = np.linalg.cholesky(A[:f, :f]) if f else np.zeros((0, 0))
        row = np.linalg.solve(L, A[:f, f]) if f else np.zeros(0)
        A[f, f] = row @ row - 0.75
        mats.append(A)
        buf = torch.from_numpy((np.tril(A) + np.triu(np.full_like(A, 9.0), 1)).T.copy()).cuda()
        dev.append(buf.t())
        rhs.append(rng.standard_normal((n, 2)))
        drhs.append(torch.from_numpy(rhs[-1].T.copy()).cuda().t())
    r, info = flame.batched("chol", dev, rhs=drhs)
    assert r == flame.FLA_SUCCESS, flame.last_error()
    for (n, f), A, d, b, db, i in zip(CASES, mats, dev, rhs, drhs, info):
        assert i == f, (n, i)
        F = to_host(d)
        assert np.array_equal(to_host(db), b), n
        assert (F[np.triu_indices(n, 1)] == 9.0).all(), n
        assert abs(F[f, f] + 0.75) < 1e-12 * np.linalg.norm(A), (n, F[f, f])
        L = np.linalg.cholesky(A[:f, :f])
        rows = np.linalg.solve(L, A[:, :f].T).T if f else np.zeros((n, 0))
        j = f // 32 * 32
        for c0, c1, r1 in ((0, j, n), (j, f, min(j + 32, n))):
            want, got = np.tril(rows[:r1, c0:c1], -c0), np.tril(F[:r1, c0:c1], -c0)
            assert np.linalg.norm(got - want) <= 1e-12 * max(1.0, np.linalg.norm(want)), (n, f, c0)
