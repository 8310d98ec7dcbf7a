"""Device memory that calls keep for later ones (until FLA_Finalize)."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

HEAD = """
import sys
sys.path.insert(0, %r)
import torch, libflame_b200 as F
F.init()
def colmajor(m, n, fill=0.0):
    return torch.full((n, m), fill, dtype=torch.float64, device="cuda").t()
def held():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]
""" % ROOT


def _run(code):
    """The last printed number of a fresh process (workspaces only grow)."""
    p = subprocess.run([sys.executable, "-c", HEAD + code], capture_output=True, text=True, timeout=300, cwd=ROOT,
                       env=dict(os.environ))
    assert p.returncode == 0, p.stderr[-2000:]
    return int(p.stdout.split()[-1])


def test_apply_q_many_columns(cuda, flame):
    """512 x 256 reflectors on 16384 columns (64 MB): the slices of the split
    products take a few times a 128 x 16384 block (16 MB), not 32 times."""
    grown = _run("""
A = torch.randn((256, 512), dtype=torch.float64, device="cuda").t()
T = colmajor(32, 256)
assert F.qr_ut(A, T) == F.FLA_SUCCESS
B = torch.randn((16384, 512), dtype=torch.float64, device="cuda").t()
assert F.apply_q_ut(A, T, B[:, :1], F.FLA_CONJ_TRANSPOSE) == F.FLA_SUCCESS
a = held()
assert F.apply_q_ut(A, T, B, F.FLA_CONJ_TRANSPOSE) == F.FLA_SUCCESS
print(a - held())
""")
    assert grown < 128 << 20, grown


def test_adjoint_scratch(cuda, flame):
    """n = 8192: the inverses of the diagonal blocks, two block columns and two
    splits' partial products, 65 MB in all, rather than 32 KB per row."""
    grown = _run("""
n = 8192
L, Lb = colmajor(n, n), colmajor(n, n, 1.0)
L.diagonal().fill_(2.0)
assert F.chol_adjoint(L[:256, :256], Lb[:256, :256]) == F.FLA_SUCCESS
a = held()
assert F.chol_adjoint(L, Lb) == F.FLA_SUCCESS
print(a - held())
""")
    assert grown < 128 << 20, grown


def test_batched_lu_short_of_memory(cuda, flame):
    """With 192 MB left for 318 MB of copies the batched LU runs in fewer CTAs instead of failing."""
    ok = _run("""
n, count = 500, 148
A = [torch.rand((n, n), dtype=torch.float64, device="cuda").t() for _ in range(count)]
A0 = [a.t().clone().t() for a in A]
P = [torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(count)]
W = [a.t().clone().t()[:8, :8] for a in A[:2]]
assert F.batched("lu", W, pivs=P[:2])[0] == F.FLA_SUCCESS
x = A[0].t().clone().t() @ A0[0][:, 0]  # the products below: loaded before memory is short
hog = torch.empty((torch.cuda.mem_get_info()[0] - (192 << 20)) // 8, dtype=torch.float64, device="cuda")
r, info = F.batched("lu", A, pivs=P)
del hog
assert r == F.FLA_SUCCESS and info == [-1] * count, F.last_error()
worst = 0.0
for a, a0, p in list(zip(A, A0, P))[::21]:
    perm = list(range(n))
    for i, q in enumerate(p.tolist()):
        perm[i], perm[i + q] = perm[i + q], perm[i]
    L = torch.tril(a, -1) + torch.eye(n, dtype=torch.float64, device="cuda")
    worst = max(worst, ((L @ torch.triu(a) - a0[perm]).norm() / (a0.norm() * n * 2.2e-16)).item())
print(int(worst < 1))
""")
    assert ok == 1
