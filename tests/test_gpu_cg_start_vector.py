"""The fused dense CG from a start vector, with a scalar part, Jacobi and a row stride: its solution, not only its
step count.  The loop scales b alone, so it starts at r0 = b / |b| - A x0 and stops at |r| <= tol |r0| + tol; a residual
r leaves an error of at most |r| / lambda_min.  Rounding: s steps add about s u cond(A) |r0| to the true residual.
Matrices: eigenvalues 0.6 .. 2.6 plus the scalar, cond <= 5."""
import pytest
import torch

import cola_gb300 as cola
from cola_gb300.linalg import cg

pytestmark = pytest.mark.gpu
U = {torch.float32: 2.0 ** -24, torch.float64: 2.0 ** -53, torch.bfloat16: 2.0 ** -24}
LAMBDA_MIN = 0.5  # of the rounded matrices, too


def _spd(n, dtype, seed):
    g = torch.Generator("cuda").manual_seed(seed)
    M = torch.randn(n, n, generator=g, device="cuda", dtype=torch.float64) / (2.0 * n ** 0.5)
    return (0.5 * (M + M.T) * 1.4 + 1.6 * torch.eye(n, device="cuda", dtype=torch.float64)).to(dtype)


# one cluster and the grid; rows resident and streamed, aligned and not; one to eight columns
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, torch.bfloat16])
@pytest.mark.parametrize("n,k", [(100, 1), (100, 2), (403, 1), (403, 2), (600, 5), (1000, 1), (1001, 8), (1500, 3),
                                 (3200, 1), (3201, 1)])
@pytest.mark.parametrize("plain", [True, False])
def test_start_vector(n, k, dtype, plain):
    if dtype == torch.float64 and n > 3000:
        n -= 1000
    vec = torch.float64 if dtype == torch.float64 else torch.float32
    wide = torch.zeros(n, n + (0 if plain else 5), device="cuda", dtype=dtype)
    wide[:, :n] = _spd(n, dtype, n)
    A = wide[:, :n]
    g = torch.Generator("cuda").manual_seed(k)
    b = torch.randn(n, k, generator=g, device="cuda", dtype=torch.float64).to(vec)
    x0 = (torch.randn(n, k, generator=g, device="cuda", dtype=torch.float64) / n ** 0.5).to(vec)
    shift = 0.0 if plain else 0.5
    op = cola.Dense(A)
    P = None
    if not plain:
        op = op + shift * cola.I_like(op)
        P = cola.Diagonal((1.0 / (A.diagonal().double() + shift)).to(vec))
    tol = 1e-10 if vec == torch.float64 else 1e-5
    x, info = cg(cola.PSD(op), b, x0=x0, P=P, tol=tol, max_iters=400)
    y, general = cg(cola.PSD(op), b, x0=x0, P=P, tol=tol, max_iters=400, allow_fused=False)
    assert info["fused"] and not general["fused"] and abs(info["iterations"] - general["iterations"]) <= 2
    A64, b64, nb = A.double(), b.double(), b.double().norm(dim=0)
    r0 = (b64 / nb - A64 @ x0.double() - shift * x0.double()).norm(dim=0)
    stop = tol * r0 + tol + info["iterations"] * 5 * U[dtype] * (1 + r0)
    for z in (x, y):
        r = (b64 - A64 @ z.double() - shift * z.double()).norm(dim=0) / nb
        assert bool((r <= stop).all())
    assert bool(((x - y).double().norm(dim=0) / nb <= 2 * stop / LAMBDA_MIN).all())
