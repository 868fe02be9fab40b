"""Which kernel takes a CSR solve with one right-hand side, at both sides of the rules: short FP32 vectors, large
matrices with and without a column window, rows of many entries (found by the kernel itself, which then
leaves the solve to the general one with x untouched).  Every route gives the general loop's solution: both
stop at |r| <= tol |r0| + tol with |r0| the residual of the scaled system, and a residual r means an error of at
most |r| / lambda_min.  The matrices are diagonally dominant by `margin`, so lambda_min >= margin."""
import pytest
import torch

import cola_gb300 as cola
from cola_gb300.linalg import cg

pytestmark = pytest.mark.gpu
MARGIN = 1.0


def _matrix(n, pairs, spread, dtype, full_row=0):
    """Symmetric, `pairs` neighbours on either side within `spread`; row 0 touches the first full_row columns."""
    g = torch.Generator("cuda").manual_seed(n + pairs)
    r = torch.arange(n, device="cuda").repeat(pairs)
    c = (r + 1 + (torch.rand(r.numel(), generator=g, device="cuda", dtype=torch.float64) * spread).long()) % n
    r, c = torch.cat([r, torch.zeros(full_row, dtype=torch.long, device="cuda")]), \
        torch.cat([c, torch.arange(full_row, device="cuda")])
    r, c = r[r != c], c[r != c]
    key = torch.unique(torch.cat([r * n + c, c * n + r]))
    r, c, i = key // n, key % n, torch.arange(n, device="cuda")
    d = torch.bincount(r, minlength=n).double() / 8 + MARGIN
    vals = torch.cat([torch.full((key.numel(),), -0.125, device="cuda", dtype=torch.float64), d])
    return cola.Sparse(vals.to(dtype), torch.cat([r, i]), torch.cat([c, i]), (n, n)), d


F32, F64 = torch.float32, torch.float64


@pytest.mark.parametrize("dtype,n,pairs,spread,full_row,kernel", [
    (F32, 8192, 2, 90, 0, "k_cg_fused"), (F32, 8193, 2, 90, 0, "k_cg_csr"), (F32, 2000, 12, 90, 0, "k_cg_csr"),
    (F64, 8192, 2, 90, 0, "k_cg_csr"),
    # above 32 MB: a window, random columns with few and with many entries; above 48 MB with long rows
    (F32, 600000, 5, 100, 0, "k_cg_csr"), (F32, 900000, 3, 900000, 0, "k_cg_csr"),
    (F32, 500000, 5, 500000, 0, "k_cg_fused"), (F64, 350000, 5, 350000, 0, "k_cg_fused"),
    (F32, 600000, 10, 60, 0, "k_cg_fused"), (F64, 120000, 15, 4000, 0, "k_cg_fused"),
    # a row of many entries in one CTA
    (F64, 5000, 2, 50, 240, "k_cg_csr"), (F64, 5000, 2, 50, 300, "k_cg_fused"), (F64, 70000, 2, 50, 70000, "k_cg_fused"),
    (F32, 40000, 2, 50, 30000, "k_cg_csr"), (F32, 40000, 2, 50, 40000, "k_cg_fused")])
@pytest.mark.parametrize("start", [False, True])
def test_route_and_solution(kernels_of, dtype, n, pairs, spread, full_row, kernel, start):
    A, d = _matrix(n, pairs, spread, dtype, full_row)
    g = torch.Generator("cuda").manual_seed(n)
    b = torch.randn(n, generator=g, device="cuda", dtype=torch.float64).to(dtype)
    x0 = torch.randn(n, generator=g, device="cuda", dtype=torch.float64).to(dtype) if start else None
    P = None if start else cola.Diagonal((1.0 / d).to(dtype))
    tol = 1e-4 if dtype == F32 else 1e-10
    (x, info), names = kernels_of(lambda: cg(cola.PSD(A), b, x0=x0, P=P, tol=tol, max_iters=400))
    ran = [k for k in ("k_cg_csr", "k_cg_fused") if any(k in name for name in names)]
    assert ran[-1:] == [kernel] and info["fused"], ran
    assert info["iterations"] - 1 < 400
    M = torch.sparse_csr_tensor(A.indptr.long(), A.indices.long(), A.values.double(), (n, n))
    r0 = 1.0 if x0 is None else float((b.double() / b.double().norm() - M @ x0.double()).norm())
    res = float((b.double() - M @ x.double()).norm() / b.double().norm())
    if x0 is None:  # the loop scales b alone: with a start vector the recursive residual is that of b/|b| - A x0
        u = 2.0 ** -24 if dtype == F32 else 2.0 ** -53
        assert res <= 2 * tol + info["iterations"] * 100 * u
    y, info2 = cg(cola.PSD(A), b, x0=x0, P=P, tol=tol, max_iters=400, allow_fused=False)
    assert abs(info["iterations"] - info2["iterations"]) <= 2
    assert float((x - y).norm() / b.norm()) <= 2 * (tol * r0 + tol) / MARGIN
