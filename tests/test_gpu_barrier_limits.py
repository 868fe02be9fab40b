"""The grid barriers of the CSR solves: the all-SM kernel for one right-hand side and the general kernel on its
cooperative grid.  With a spin limit of one poll a CTA that arrives before the last one gives up (always the case on a
grid of 152 CTAs and more), the call returns COLAGB_ERR_TIMEOUT with x as it was, and the next call solves normally.
No GPU fault, trap or endless loop is involved.

The matrix is tridiagonal (3, -1): cond 5, so that 60 steps contract the error by 0.39 each, to FP32 rounding; the
residual left is that of the steps' roundings, about 60 u cond."""
import ctypes as C

import pytest
import torch

import cola_gb300 as cola
from cola_gb300 import _capi
from cola_gb300.lowering import Lowered

pytestmark = pytest.mark.gpu


def _solve(op, B, spin_limit):
    lib = _capi.load()
    low = Lowered(op)
    n, k = B.shape
    X = torch.zeros_like(B)
    prm = _capi.CgParams(tol=0.0, max_iters=60, check_every=16, allow_fused=1, graph=0, spin_limit=spin_limit)
    res, nb = _capi.CgResult(), C.c_size_t()
    _capi.check(lib.colagb_cg_workspace_bytes(low.handle, None, k, C.byref(nb)), "ws")
    ws = torch.empty(nb.value, dtype=torch.uint8, device="cuda")
    st = lib.colagb_cg_solve(low.handle, None, B.data_ptr(), k, X.data_ptr(), k, k, C.byref(prm), None, ws.data_ptr(),
                             nb.value, C.byref(res), _capi.stream_ptr(B.device))
    torch.cuda.synchronize()
    return st, res, X


# one right-hand side (k_cg_csr), and more than 32 MB with several (k_cg_fused on the cooperative grid)
@pytest.mark.parametrize("n,k", [(60000, 1), (1500000, 2)])
def test_barrier_gives_up_and_the_next_call_solves(n, k):
    i = torch.arange(n, device="cuda")
    vals = torch.cat([torch.full((n,), 3.0, device="cuda"), torch.full((2 * n - 2,), -1.0, device="cuda")])
    A = cola.Sparse(vals, torch.cat([i, i[1:], i[:-1]]), torch.cat([i, i[:-1], i[1:]]), (n, n))
    op = cola.PSD(A)
    B = torch.randn(n, k, generator=torch.Generator("cuda").manual_seed(k), device="cuda")
    st, res, X = _solve(op, B, spin_limit=1)
    assert res.fused == 1 and st == _capi.ERR_TIMEOUT and res.status == _capi.ERR_TIMEOUT
    assert b"timed out" in _capi.load().colagb_last_error()
    assert k > 1 or float(X.abs().max()) == 0.0
    st, res, X = _solve(op, B, spin_limit=0)
    assert st == _capi.OK and res.status == 0 and res.iterations == 60 and res.fused == 1
    X64 = X.double()
    R = B.double() - 3.0 * X64
    R[1:] += X64[:-1]
    R[:-1] += X64[1:]
    assert float((R.norm(dim=0) / B.double().norm(dim=0)).max()) <= 4 * 60 * 5 * 2.0 ** -24
