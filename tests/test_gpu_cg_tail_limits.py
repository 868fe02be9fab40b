"""Where a step of the generic CG loop ends in one cluster launch and where in three, at both sides of the limits
for each kind of column count, type and scalar part.  The operator is diagonal (1 .. 2, plus the scalar part), so
the solution is known: cond 2 contracts the error by 0.18 a step, and the residual the loop stops at, tol |r0| + tol
with |r0| = 1, bounds the error by 2 tol |b| / 1 plus the 30 steps' roundings."""
import pytest
import torch

import cola_gb300 as cola
from cola_gb300.linalg import cg

pytestmark = pytest.mark.gpu
F32, F64 = torch.float32, torch.float64


# entries (of 1024) up to which a block takes one launch
@pytest.mark.parametrize("dtype,k,scalar,limit", [
    (F32, 1, False, 180), (F32, 1, True, 276), (F32, 8, False, 320), (F32, 16, False, 512), (F32, 16, True, 512),
    (F32, 3, False, 128), (F32, 3, True, 224), (F32, 12, False, 256), (F32, 20, False, 320), (F32, 33, False, 512),
    (F64, 1, False, 24), (F64, 2, False, 32), (F64, 3, False, 48), (F64, 1, True, 48)])
@pytest.mark.parametrize("jacobi", [False, True])
def test_limits(kernels_of, dtype, k, scalar, limit, jacobi):
    u = 2.0 ** -24 if dtype == F32 else 2.0 ** -53
    tol = 1e-5 if dtype == F32 else 1e-11
    for n, one in ((limit * 1024 // k, True), (limit * 1024 // k + 1, False)):
        d = torch.linspace(1.0, 2.0, n, device="cuda", dtype=F64)
        op = cola.Diagonal(d.to(dtype))
        if scalar:
            op = op + 0.5 * cola.I_like(op)
        b = torch.randn(n, k, generator=torch.Generator("cuda").manual_seed(k), device="cuda", dtype=F64).to(dtype)
        P = cola.Diagonal(torch.linspace(1.0, 0.9, n, device="cuda", dtype=F64).to(dtype)) if jacobi else None
        (x, info), names = kernels_of(lambda: cg(cola.PSD(op), b, P=P, tol=tol, max_iters=100))
        assert any("k_cg_tail" in name for name in names) == one
        assert not info["fused"] and info["iterations"] - 1 <= 30
        exact = b.double() / (d.to(dtype).double() + (0.5 if scalar else 0.0))[:, None]
        err = (x.double() - exact).norm(dim=0) / b.double().norm(dim=0)
        assert float(err.max()) <= 2 * tol + 30 * 10 * u
