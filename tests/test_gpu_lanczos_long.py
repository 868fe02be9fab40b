"""Lanczos and Arnoldi at both sides of the sizes from which every pass over the basis is a launch of its own:
the kernels that run, and the identities of the exact process (orthonormal basis, A Q = Q T + beta q e^T).

Tolerances: with u the unit roundoff, |A| = 2 and n-term sums whose rounding grows like sqrt(n) at worst here,
two Gram-Schmidt passes leave |Q^T Q - I| and the recurrence within 32 sqrt(n) u |A|."""
import pytest
import torch

import cola_gb300 as cola
from cola_gb300.linalg.arnoldi import run_arnoldi
from cola_gb300.linalg.lanczos import run_lanczos

pytestmark = pytest.mark.gpu
U = {torch.float32: 2.0 ** -24, torch.float64: 2.0 ** -53}
F32, F64 = torch.float32, torch.float64


def _problem(n, bs, dtype):
    g = torch.Generator("cuda").manual_seed(n + bs)
    d = (1.0 + torch.rand(n, generator=g, device="cuda", dtype=F64)).to(dtype)
    return cola.ops.Diagonal(d), d.double(), torch.randn(n, bs, generator=g, device="cuda", dtype=F64).to(dtype)


@pytest.mark.parametrize("dtype,n,bs,passes", [
    (F32, 109226, 3, False), (F32, 109227, 3, True), (F32, 46812, 7, True), (F32, 9930, 33, True), (F32, 327683, 1, True),
    (F32, 2521, 130, True), (F32, 16385, 20, True), (F32, 1300, 260, True), (F32, 81924, 4, False), (F32, 200001, 7, True),
    (F64, 110000, 10, False), (F64, 110001, 10, True), (F64, 33334, 33, True), (F64, 1100001, 1, True),
    (F64, 4232, 260, True), (F64, 8462, 130, False)])
def test_lanczos(kernels_of, dtype, n, bs, passes):
    op, d, V = _problem(n, bs, dtype)
    m = 9
    res, names = kernels_of(lambda: run_lanczos(op, V, m, 0.0))
    assert any("k_lz_project<" in name for name in names) == passes and res.iters == m
    Q, beta = res.basis[1:].double(), res.subdiag[:, 1:].double()  # (m + 1, n, bs), the last one not normalised
    Q[m] /= beta[:, m - 1]
    tol = 32 * n ** 0.5 * U[dtype] * 2
    G = torch.einsum("inb,jnb->bij", Q, Q)
    assert float((G - torch.eye(m + 1, device="cuda", dtype=F64)).abs().max()) <= tol
    for i in range(m):
        r = d[:, None] * Q[i] - res.diag[:, i].double() * Q[i] - beta[:, i] * Q[i + 1]
        if i:
            r -= beta[:, i - 1] * Q[i - 1]
        assert float(r.norm(dim=0).max()) <= tol


@pytest.mark.parametrize("dtype,n,bs,passes", [(F32, 366667, 3, True), (F32, 366666, 3, False), (F32, 275001, 4, True),
                                               (F64, 550001, 2, True), (F64, 33334, 33, True), (F64, 1100001, 1, True)])
def test_arnoldi(kernels_of, dtype, n, bs, passes):
    op, d, V = _problem(n, bs, dtype)
    m = 7
    (Q, H, steps), names = kernels_of(lambda: run_arnoldi(op, V, m, 0.0))
    assert any("k_lz_project<" in name for name in names) == passes and steps == m
    Q, H = Q.double(), H.double()
    tol = 32 * n ** 0.5 * U[dtype] * 2
    G = Q.transpose(1, 2) @ Q
    assert float((G - torch.eye(m + 1, device="cuda", dtype=F64)).abs().max()) <= tol
    assert float((d[:, None] * Q[:, :, :m] - Q @ H).norm(dim=1).max()) <= tol
