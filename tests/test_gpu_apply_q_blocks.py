"""FLA_Apply_Q_UT by super-blocks: orders around the 128-column super-blocks
and their odd ends, T blocks that do not divide 128, reflectors off the
16-byte grid, both directions, against the oracle's block-by-block product.

Tolerance: Q^T B and Q B are products of orthogonal factors, so both sides are
within about (columns) eps of the exact one; 1e-12 normwise as in the other
parity tests."""
import numpy as np
import pytest

from conftest import rel_fro, seeded, to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,b,nrhs", [(128, 128, 32, 8), (129, 129, 32, 1), (260, 127, 32, 9), (300, 130, 32, 33),
                                        (257, 257, 32, 7), (1400, 385, 32, 70), (2101, 131, 32, 2), (700, 300, 24, 20),
                                        (200, 77, 5, 3), (331, 200, 33, 12), (420, 201, 100, 5), (300, 140, 71, 4)])
def test_apply_q_blocks(cuda, flame, oracle, m, n, b, nrhs):
    rng = seeded(m + 7 * n + b)
    A = rng.standard_normal((m, n))
    QR, T = oracle.qr_ut(A, b)
    B = rng.standard_normal((m, nrhs))
    Ad, Td = to_dev(cuda, QR), to_dev(cuda, T)
    Bd = to_dev(cuda, B)
    assert flame.apply_q_ut(Ad, Td, Bd) == flame.FLA_SUCCESS, flame.last_error()
    assert rel_fro(to_host(Bd), oracle.apply_qt(QR, T, B)) < 1e-12
    # Q B, from the oracle's Q^T applied to the identity
    Q = oracle.apply_qt(QR, T, np.eye(m)).T
    Bd = to_dev(cuda, B)
    assert flame.apply_q_ut(Ad, Td, Bd, flame.FLA_NO_TRANSPOSE) == flame.FLA_SUCCESS, flame.last_error()
    assert rel_fro(to_host(Bd), Q @ B) < 1e-12
