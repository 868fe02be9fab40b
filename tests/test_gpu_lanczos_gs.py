"""The orthogonalisation kernels of Lanczos and Arnoldi over block widths, odd sizes and both types, by
the two identities of the exact process: the basis is orthonormal and A Q = Q T + beta q e^T.

Tolerances: with u the unit roundoff, |A| = 2 and n-term sums whose rounding grows like sqrt(n) at worst
here, two Gram-Schmidt passes leave |Q^T Q - I| and the recurrence within 32 sqrt(n) u |A|."""
import pytest
import torch

import cola_gb300 as cola
from cola_gb300.linalg.arnoldi import run_arnoldi
from cola_gb300.linalg.lanczos import run_lanczos

pytestmark = pytest.mark.gpu
U = {torch.float32: 2.0 ** -24, torch.float64: 2.0 ** -53}
SHAPES = [(6, 1), (37, 1), (130, 1), (4096, 1), (5001, 1), (20000, 1), (50, 3), (64, 4), (333, 5), (1000, 13), (4000, 16),
          (777, 31), (600, 32), (500, 36), (257, 33), (300, 64), (200, 130), (96, 300)]


def _problem(n, bs, dtype):
    g = torch.Generator("cuda").manual_seed(n + bs)
    d = 1.0 + torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    d, V = d.to(dtype), torch.randn(n, bs, generator=g, device="cuda", dtype=torch.float64).to(dtype)
    return cola.ops.Diagonal(d), d.double(), V


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("n,bs", SHAPES)
def test_lanczos_identities(n, bs, dtype):
    op, d, V = _problem(n, bs, dtype)
    m = min(9, n - 1)
    res = run_lanczos(op, V, m, 0.0)
    assert res.iters == m
    Q = res.basis[1:].double()  # (m + 1, n, bs), the last one not normalised
    beta = res.subdiag[:, 1:].double()
    Q[m] /= beta[:, m - 1]
    tol = 32 * n ** 0.5 * U[dtype] * 2
    G = torch.einsum("inb,jnb->bij", Q, Q)
    assert float((G - torch.eye(m + 1, device="cuda", dtype=torch.float64)).abs().max()) <= tol
    for i in range(m):
        r = d[:, None] * Q[i] - res.diag[:, i].double() * Q[i] - beta[:, i] * Q[i + 1]
        if i:
            r -= beta[:, i - 1] * Q[i - 1]
        assert float(r.norm(dim=0).max()) <= tol
    assert float(res.basis[0].abs().max()) == 0.0


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("n,bs", [(37, 1), (5001, 1), (333, 5), (4000, 16), (257, 33)])
def test_arnoldi_identities(n, bs, dtype):
    g = torch.Generator("cuda").manual_seed(n)
    A = torch.randn(n, n, generator=g, device="cuda", dtype=torch.float64).div_(n ** 0.5).to(dtype)
    V = torch.randn(n, bs, generator=g, device="cuda", dtype=torch.float64).to(dtype)
    m = 9
    Q, H, steps = run_arnoldi(cola.ops.Dense(A), V, m, 0.0)
    assert steps == m
    Q, H = Q.double(), H.double()
    tol = 32 * n ** 0.5 * U[dtype] * 2
    G = Q.transpose(1, 2) @ Q
    assert float((G - torch.eye(m + 1, device="cuda", dtype=torch.float64)).abs().max()) <= tol
    assert float((A.double() @ Q[:, :, :m] - Q @ H).norm(dim=1).max()) <= tol


def test_unfilled_slots_read_zero():
    n = 64
    d = torch.ones(n, device="cuda", dtype=torch.float64)
    d[:3] = torch.tensor([2.0, 3.0, 4.0], device="cuda")
    V = torch.zeros(n, 1, device="cuda", dtype=torch.float64)
    V[:4] = 1.0  # four distinct eigenvalues: an invariant subspace after four steps
    res = run_lanczos(cola.ops.Diagonal(d), V, 40, 1e-8)
    assert res.iters <= 5
    assert float(res.basis[res.i_final + 1:].abs().max()) == 0.0 and float(res.basis[0].abs().max()) == 0.0
