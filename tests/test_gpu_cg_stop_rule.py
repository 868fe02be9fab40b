"""The stop rule of the fused CG schedules at the ends of its range: steps go on while |r| > tol |r0| + tol,
so a negative tolerance takes max_iters steps and an infinite one none, as in the general loop."""
import math

import pytest
import torch

import cola_gb300 as cola
from cola_gb300.linalg import cg

pytestmark = pytest.mark.gpu


def _dense(n, dtype):
    g = torch.Generator("cuda").manual_seed(n)
    M = torch.randn(n, n, generator=g, device="cuda", dtype=torch.float64) / (2.0 * n ** 0.5)
    return cola.Dense((0.5 * (M + M.T) * 1.4 + 1.6 * torch.eye(n, device="cuda", dtype=torch.float64)).to(dtype))


def _tridiagonal(n, dtype):
    i = torch.arange(n, device="cuda")
    rows = torch.cat([i, i[1:], i[:-1]])
    cols = torch.cat([i, i[:-1], i[1:]])
    vals = torch.cat([torch.full((n,), 3.0, device="cuda"), torch.full((2 * n - 2,), -1.0, device="cuda")])
    return cola.Sparse(vals.to(dtype), rows, cols, (n, n))


# one cluster, the grid, several columns; few and many rows a CTA of the CSR schedule
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("make,n,k", [(_dense, 100, 1), (_dense, 1000, 1), (_dense, 600, 3), (_tridiagonal, 500, 1),
                                      (_tridiagonal, 80000, 1)])
@pytest.mark.parametrize("tol,steps", [(-1.0, 12), (-1e-3, 12), (0.0, 12), (math.inf, 0), (math.nan, 0)])
def test_tolerance_range(make, n, k, dtype, tol, steps):
    op = cola.PSD(make(n, dtype))
    b = torch.randn(n, k, generator=torch.Generator("cuda").manual_seed(k), device="cuda", dtype=torch.float64).to(dtype)
    b = b[:, 0].contiguous() if k == 1 else b
    x, info = cg(op, b, tol=tol, max_iters=12)
    y, general = cg(op, b, tol=tol, max_iters=12, allow_fused=False)
    assert info["fused"] and not general["fused"]
    assert info["iterations"] == general["iterations"] == steps + 1
    # a step contracts the error by (sqrt(c) - 1) / (sqrt(c) + 1) <= 0.46 at cond c <= 7.3; both loops round
    # each of the 12 steps' vectors by a few u, times cond
    u = 2.0 ** -24 if dtype == torch.float32 else 2.0 ** -53
    assert float((x - y).norm()) <= 12 * 8 * 7.3 * u * max(float(y.norm()), 1e-30) * (1 if steps else 0)
