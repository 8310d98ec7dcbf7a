"""FLA_B200_batched_tune / FLA_B200_batched_nb: the FP64 kernels have one panel
width, which tuning leaves; the FP32 ones are correct at the widths it chooses.
Bar for FP32: the backward error of n steps in 24-bit arithmetic, 4 n eps."""
import ctypes as C

import numpy as np
import pytest

from conftest import seeded, spd

pytestmark = pytest.mark.gpu

ORDERS = (16, 48, 100, 200, 400)


@pytest.mark.parametrize("lu", [0, 1])
def test_fp64_width_is_fixed(cuda, flame, lu):
    L = flame.lib()
    assert [L.FLA_B200_batched_nb(lu, 1, n) for n in ORDERS] == [32] * 5
    times = (C.c_double * 20)()
    assert L.FLA_B200_batched_tune(lu, 1, 2, times) == flame.FLA_SUCCESS, flame.last_error()
    t = np.array(times).reshape(5, 4)
    assert (t > 0).all() and (t == t[:, :1]).all()
    assert [L.FLA_B200_batched_nb(lu, 1, n) for n in ORDERS] == [32] * 5


@pytest.mark.parametrize("kind", ["chol", "lu"])
def test_fp32_at_tuned_widths(cuda, flame, kind):
    torch = cuda
    times = (C.c_double * 20)()
    assert flame.lib().FLA_B200_batched_tune(int(kind == "lu"), 0, 4, times) == flame.FLA_SUCCESS, flame.last_error()
    assert all(t > 0 for t in times)
    rng = seeded(9)
    mats = [(spd(rng, n) if kind == "chol" else rng.uniform(-1, 1, (n, n))).astype(np.float32) for n in ORDERS]
    dev = [torch.from_numpy(A.T.copy()).cuda().t() for A in mats]
    piv = [torch.zeros(n, dtype=torch.int32, device="cuda") for n in ORDERS]
    r, info = flame.batched(kind, dev, pivs=piv if kind == "lu" else None, f32=True)
    assert r == flame.FLA_SUCCESS and info == [-1] * 5, (info, flame.last_error())
    for n, A, d, p in zip(ORDERS, mats, dev, piv):
        X, P = d.cpu().numpy().astype(np.float64), A.astype(np.float64)
        if kind == "chol":
            L, U = np.tril(X), np.tril(X).T
        else:
            for i, q in enumerate(p.cpu().numpy()):
                P[[i, i + q]] = P[[i + q, i]]
            L, U = np.tril(X, -1) + np.eye(n), np.triu(X)
        bound = 4 * n * 2.0 ** -23 * np.linalg.norm(np.abs(L) @ np.abs(U))
        assert np.linalg.norm(L @ U - P) <= bound, n
