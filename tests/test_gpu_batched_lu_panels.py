"""FLA_LU_piv_batched at the edges of its 32-column panels, update tiles and the
256 / 512-thread split, with padded leading dimensions and up to eight
right-hand sides, each matrix against the oracle's FLA_LU_piv.

Bars as in the other batched tests: pivots identical, factors within 1e-12
normwise, solutions within 1e-11 of the oracle's; a singular matrix keeps its
right-hand side and reports its first zero column."""
import numpy as np
import pytest

from conftest import rel_fro, seeded, to_dev, to_host

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 31, 32, 33, 63, 64, 65, 95, 97, 128, 159, 255, 256, 257, 287, 289, 480, 481, 497, 511, 512]


@pytest.mark.parametrize("nrhs,pad", [(0, 0), (1, 3), (8, 1)])
def test_panels_and_tiles(cuda, flame, oracle, nrhs, pad):
    torch = cuda
    rng = seeded(71 + nrhs)
    mats = [rng.uniform(-1, 1, (n, n)) for n in SIZES]
    sing = SIZES.index(97)
    mats[sing][:, 40] = 0.0
    ties = SIZES.index(65)
    mats[ties][:, 0] = 0.25
    dev = []
    for A in mats:
        n = A.shape[0]
        buf = torch.full((n, n + pad), float("nan"), dtype=torch.float64, device="cuda")  # rows: columns of A
        buf[:, :n] = torch.from_numpy(A.T.copy())
        dev.append(buf.t()[:n, :])
    pivs = [torch.zeros(n, dtype=torch.int32, device="cuda") for n in SIZES]
    rhs = [rng.standard_normal((n, nrhs)) for n in SIZES] if nrhs else None
    drhs = [to_dev(torch, b) for b in rhs] if nrhs else None
    if nrhs == 1:  # a one-column view has no second stride of its own
        drhs = [torch.empty_strided((n, 1), (1, n), dtype=torch.float64, device="cuda").copy_(torch.from_numpy(b))
                for n, b in zip(SIZES, rhs)]
    r, info = flame.batched("lu", dev, pivs=pivs, rhs=drhs)
    assert r == flame.FLA_SUCCESS, flame.last_error()
    for i, A in enumerate(mats):
        LUo, po, ro = oracle.lu_piv(A)
        assert info[i] == ro, (SIZES[i], info[i], ro)
        assert np.array_equal(pivs[i].cpu().numpy(), po), SIZES[i]
        assert rel_fro(to_host(dev[i]), LUo) < 1e-12, SIZES[i]
        if nrhs and ro == -1:
            assert rel_fro(to_host(drhs[i]), oracle.lu_piv_solve(LUo, po, rhs[i])) < 1e-11, SIZES[i]
        elif nrhs:
            assert np.array_equal(to_host(drhs[i]), rhs[i])
