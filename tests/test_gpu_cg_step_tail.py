"""The generic CG loop's step as one cluster launch (k_cg_tail): column counts with and without the shuffle
sums, blocks at both sides of its size limits, Jacobi, and the scalar part of a sum folded into it.

The operator is a Kronecker product of two factors with eigenvalues 1..5 (cond 25).  From a zero start the
recursive residual stops at tol |r0| + tol with |r0| = 1, and s steps add at most about s u cond(A) to the
true one.  A preconditioner written as a product takes the separate launches: the same number of steps."""
import pytest
import torch

import cola_gb300 as cola
from cola_gb300.linalg import cg

pytestmark = pytest.mark.gpu
U = {torch.float32: 2.0 ** -24, torch.float64: 2.0 ** -53}
TOL = {torch.float32: 1e-5, torch.float64: 1e-11}


def _factor(n, dtype, seed):
    g = torch.Generator().manual_seed(seed)
    Q = torch.linalg.qr(torch.randn(n, n, generator=g, dtype=torch.float64))[0]
    return ((Q * torch.linspace(1.0, 5.0, n, dtype=torch.float64)) @ Q.T).to("cuda", dtype)


SIZES = [(torch.float32, 3, 5, 1), (torch.float32, 31, 33, 2), (torch.float32, 31, 33, 3), (torch.float32, 64, 16, 32),
         (torch.float32, 32, 31, 33), (torch.float32, 96, 80, 68), (torch.float32, 96, 80, 69), (torch.float32, 32, 32, 512),
         (torch.float32, 16, 32, 513), (torch.float64, 3, 5, 1), (torch.float64, 31, 33, 4), (torch.float64, 96, 80, 6),
         (torch.float64, 96, 80, 7), (torch.float64, 8, 12, 512)]


@pytest.mark.parametrize("kind", ["plain", "jacobi", "sum", "sum_first"])
@pytest.mark.parametrize("dtype,n1,n2,k", SIZES)
def test_step_tail(dtype, n1, n2, k, kind):
    F, G = _factor(n1, dtype, n1), _factor(n2, dtype, n2 + 100)
    n = n1 * n2
    b = torch.randn(n, k, generator=torch.Generator().manual_seed(k), dtype=torch.float64).to("cuda", dtype)
    K = cola.Kronecker(cola.Dense(F), cola.Dense(G))
    shift = 0.5 if kind.startswith("sum") else 0.0
    op = {"sum": lambda: K + shift * cola.I_like(K), "sum_first": lambda: shift * cola.I_like(K) + K}.get(kind, lambda: K)()
    d = 1.0 / (torch.kron(F.diagonal(), G.diagonal()) + shift)
    P = cola.Diagonal(d) if kind == "jacobi" else None
    x, info = cg(cola.PSD(op), b, P=P, tol=TOL[dtype], max_iters=400)
    assert not info["fused"] and info["iterations"] - 1 <= 200
    X = x.double().reshape(n1, n2, k)
    AX = torch.einsum("ij,jbk->ibk", F.double(), torch.einsum("ab,jbk->jak", G.double(), X)).reshape(n, k) + shift * x.double()
    rel = ((b.double() - AX).norm(dim=0) / b.double().norm(dim=0)).max()
    assert float(rel) <= 2 * TOL[dtype] + 200 * 25 * U[dtype]
    one = cola.Diagonal(torch.ones_like(d))
    general = cola.Product(cola.Diagonal(d), one) if kind == "jacobi" else cola.Product(one, one)
    y, info2 = cg(cola.PSD(op), b, P=general, tol=TOL[dtype], max_iters=400)
    assert abs(info["iterations"] - info2["iterations"]) <= 2


@pytest.mark.parametrize("dtype,n,k,fused", [(torch.float32, 2150, 8, True), (torch.float32, 2250, 8, False),
                                             (torch.float32, 2251, 5, False), (torch.bfloat16, 2400, 5, False),
                                             (torch.float64, 1201, 8, False)])
@pytest.mark.parametrize("form", ["plain", "jacobi_shift"])
def test_dense_columns_that_do_not_fit(dtype, n, k, fused, form):
    """Several columns beyond the one-exchange kernel's shared memory: the generic loop, without a graph.
    Cond 5 (BF16 storage moves the eigenvalues by less than 5 * 2^-8 * 2)."""
    vec = torch.float64 if dtype == torch.float64 else torch.float32
    A = _factor(n, dtype, 7)
    A = torch.tril(A) + torch.tril(A, -1).T
    b = torch.randn(n, k, generator=torch.Generator().manual_seed(k), dtype=torch.float64).to("cuda", vec)
    D, shift, P = cola.Dense(A), 0.0, None
    op = D
    if form == "jacobi_shift":
        shift, op = 0.25, D + 0.25 * cola.I_like(D)
        P = cola.Diagonal((1.0 / (A.diagonal().double() + 0.25)).to(vec))
    tol = TOL[vec]
    x, info = cg(cola.PSD(op), b, P=P, tol=tol, max_iters=400)
    assert info["fused"] == fused and not info["graph"] and info["iterations"] - 1 <= 200
    R = b.double() - A.double() @ x.double() - shift * x.double()
    assert float((R.norm(dim=0) / b.double().norm(dim=0)).max()) <= 2 * tol + 200 * 25 * U[vec]
    y, info2 = cg(cola.PSD(op), b, P=P, tol=tol, max_iters=400, allow_fused=False)
    assert abs(info["iterations"] - info2["iterations"]) <= 2
    assert len(info["errors"]) in (info["iterations"] - 1, info["iterations"])
