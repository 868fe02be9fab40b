"""The fused CG schedules of one Dense operator (one exchange per step) and of one CSR operator (column
windows, or gathers where the columns spread): sizes at the edges of their partitions, rows resident or
streamed, aligned or not, several right-hand sides, shift, Jacobi and a start vector.

Each solution's true residual is checked in FP64.  From a zero start the recursive residual stops at
tol |r0| + tol with |r0| = 1; a solve of s steps adds at most about s u cond(A) to the true one, with
cond <= 30 and s <= 200 here.  The general loop has to take the same number of steps, from a start vector
too (whose stop threshold is that of the unscaled A x0)."""
import pytest
import torch

import cola_gb300 as cola
from cola_gb300.linalg import cg

pytestmark = pytest.mark.gpu
U = {torch.float32: 2.0 ** -24, torch.float64: 2.0 ** -53, torch.bfloat16: 2.0 ** -24}
TOL = {torch.float32: 1e-5, torch.bfloat16: 1e-5, torch.float64: 1e-11}


def _check(matvec64, op, b, dtype, P=None, x0=None, fused=True):
    x, info = cg(op, b, x0=x0, P=P, tol=TOL[dtype], max_iters=400)
    assert info["fused"] == fused and info["iterations"] - 1 <= 200
    B, X = b.double().reshape(b.shape[0], -1), x.double().reshape(b.shape[0], -1)
    rel = ((B - matvec64(X)).norm(dim=0) / B.norm(dim=0)).max()
    if x0 is None:
        assert float(rel) <= 2 * TOL[dtype] + 200 * 30 * U[dtype]
    y, info2 = cg(op, b, x0=x0, P=P, tol=TOL[dtype], max_iters=400, allow_fused=False)
    assert abs(info["iterations"] - info2["iterations"]) <= 2
    assert len(info["errors"]) == info["iterations"] - 1 or len(info["errors"]) == info["iterations"]


def _spd(n, dtype, seed):
    g = torch.Generator("cuda").manual_seed(seed)
    M = torch.randn(n, n, generator=g, device="cuda", dtype=torch.float64) / (2.0 * n ** 0.5)
    return (0.5 * (M + M.T) * 1.4 + 1.6 * torch.eye(n, device="cuda", dtype=torch.float64)).to(dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, torch.bfloat16])
@pytest.mark.parametrize("n,k", [(8, 1), (9, 2), (15, 1), (16, 1), (64, 3), (151, 1), (153, 1), (200, 8), (300, 5), (513, 2),
                                 (700, 1), (1001, 4), (1500, 1), (2050, 1), (3001, 3)])
def test_dense(n, k, dtype):
    if dtype == torch.float64 and n > 2100:
        n = 2101
    A = _spd(n, dtype, n)
    b = torch.randn(n, k, generator=torch.Generator("cuda").manual_seed(k), device="cuda", dtype=torch.float64)
    b = b.to(torch.float64 if dtype == torch.float64 else torch.float32)
    op = cola.PSD(cola.Dense(A))
    _check(lambda X: A.double() @ X, op, b[:, 0] if k == 1 else b, dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_dense_shift_jacobi_start_and_row_stride(dtype):
    n, k = 403, 2
    wide = torch.zeros(n, n + 5, device="cuda", dtype=dtype)
    wide[:, :n] = _spd(n, dtype, 3)
    A = wide[:, :n]
    g = torch.Generator("cuda").manual_seed(4)
    b = torch.randn(n, k, generator=g, device="cuda", dtype=torch.float64).to(dtype)
    x0 = torch.randn(n, k, generator=g, device="cuda", dtype=torch.float64).to(dtype)
    D = cola.Dense(A)
    op = cola.PSD(D + 0.5 * cola.I_like(D))
    P = cola.Diagonal(1.0 / (A.diagonal() + 0.5))
    _check(lambda X: A.double() @ X + 0.5 * X, op, b, dtype, P=P, x0=x0)


def _sparse(n, spread, dtype, seed):
    """Symmetric, diagonally dominant, about seven entries a row: neighbours near (spread small) or anywhere."""
    g = torch.Generator("cuda").manual_seed(seed)
    r = torch.arange(n, device="cuda").repeat(3)
    hop = 1 + (torch.rand(3 * n, generator=g, device="cuda", dtype=torch.float64) * spread).long()
    c = (r + hop) % n
    keep = r != c
    key = torch.unique(torch.cat([r[keep] * n + c[keep], c[keep] * n + r[keep]]))
    r, c = key // n, key % n
    w = 0.5 + 0.5 * torch.cos((r * c % 1000).double())  # symmetric in r, c
    d = torch.zeros(n, device="cuda", dtype=torch.float64).index_add_(0, r, w) + 0.5
    rows, cols = torch.cat([r, torch.arange(n, device="cuda")]), torch.cat([c, torch.arange(n, device="cuda")])
    return cola.Sparse(torch.cat([-w, d]).to(dtype), rows, cols, (n, n))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, torch.bfloat16])
@pytest.mark.parametrize("n,spread", [(1, 1), (31, 3), (33, 5), (1000, 40), (4865, 4865), (70001, 300), (70001, 70001)])
def test_csr(n, spread, dtype):
    A = _sparse(n, spread, dtype, n + spread)
    ip, ix, v = A.indptr.long(), A.indices.long(), A.values.double()
    M = torch.sparse_csr_tensor(ip, ix, v, (n, n))
    g = torch.Generator("cuda").manual_seed(n)
    vec = torch.float64 if dtype == torch.float64 else torch.float32
    b = torch.randn(n, generator=g, device="cuda", dtype=torch.float64).to(vec)
    rows = torch.repeat_interleave(torch.arange(n, device="cuda"), ip[1:] - ip[:-1])
    diag = v[rows == ix]
    _check(lambda X: M @ X, cola.PSD(A), b, dtype, P=cola.Diagonal((1.0 / diag).to(vec)))
    x0 = torch.randn(n, generator=g, device="cuda", dtype=torch.float64).to(vec)
    _check(lambda X: M @ X + 0.25 * X, cola.PSD(A + 0.25 * cola.I_like(A)), b, dtype, x0=x0)
