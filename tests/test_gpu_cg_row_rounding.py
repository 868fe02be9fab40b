"""Rounding of the fused dense CG's FP32 row sums, seen alone.

The columns of A come in equal pairs and x0 has opposite entries for them, so A x0 is zero exactly and the first
residual, b / |b| - A x0, holds e_0 and the rounding errors of the row sums; its norm is the history's
first entry.  The errors' norm may not exceed that of the plain order the row kernels follow or improve on
(lane l of 32 takes the quads l, l + 32, ... of a row, adds a quad's four products to each other and
then to its sum, and the lanes are added in a tree), formed here step by step in FP32 on the same
numbers.  Two orders of equal expectation differ by chance: each of the n rows' squared errors varies
by about its own size, so the ratio of two norms over s problems of n rows has a relative deviation of
about sqrt(1 / (n s)), 1.1 % at n = 1024 and s = 8; the test allows 5 %."""
import ctypes as C

import pytest
import torch

import cola_gb300 as cola
from cola_gb300 import _capi
from cola_gb300.lowering import Lowered

pytestmark = pytest.mark.gpu
BIG = 2.0 ** 30  # of x0: the errors, about 2^-24 BIG, beside |e_0| = 1


def _problem(n, seed):
    g = torch.Generator("cuda").manual_seed(seed)
    order = torch.randperm(n, generator=g, device="cuda")
    a, b = order[: n // 2], order[n // 2:]
    half = torch.randn(n, n // 2, generator=g, device="cuda")
    x = BIG * torch.randn(n // 2, generator=g, device="cuda")
    A, x0 = torch.empty(n, n, device="cuda"), torch.empty(n, device="cuda")
    A[:, a], A[:, b] = half, half
    x0[a], x0[b] = x, -x
    return A, x0


def _first_residual(A, x0):
    lib, n = _capi.load(), A.shape[0]
    low = Lowered(cola.PSD(cola.Dense(A)))
    b = torch.zeros(n, 1, device="cuda")
    b[0] = 1.0
    X, hist = x0[:, None].clone(), torch.zeros(1, device="cuda")
    prm = _capi.CgParams(tol=0.0, max_iters=0, check_every=16, allow_fused=1, graph=0, spin_limit=0)
    res, nb = _capi.CgResult(), C.c_size_t()
    _capi.check(lib.colagb_cg_workspace_bytes(low.handle, None, 1, C.byref(nb)), "ws")
    ws = torch.empty(nb.value, dtype=torch.uint8, device="cuda")
    _capi.check(lib.colagb_cg_solve(low.handle, None, b.data_ptr(), 1, X.data_ptr(), 1, 1, C.byref(prm), hist.data_ptr(),
                                    ws.data_ptr(), nb.value, C.byref(res), _capi.stream_ptr(b.device)), "cg")
    assert res.fused == 1
    return float(hist[0])


def _plain_order(A, x0):
    n = A.shape[0]
    pad = -n % 128
    A, x = torch.nn.functional.pad(A, (0, pad)).double(), torch.nn.functional.pad(x0, (0, pad)).double()
    P = (A * x).reshape(n, -1, 32, 4)  # products of FP32 numbers, exact in FP64
    f32 = lambda v: v.float().double()  # noqa: E731
    lane = torch.zeros(n, 32, dtype=torch.float64, device="cuda")
    for u in range(P.shape[1]):
        s = f32(P[:, u, :, 0])
        for e in (1, 2, 3):
            s = f32(s + P[:, u, :, e])
        lane = f32(lane + s)
    while lane.shape[1] > 1:
        h = lane.shape[1] // 2
        lane = f32(lane[:, :h] + lane[:, h:])
    r = lane[:, 0]
    r[0] -= 1.0
    return float(r.norm())


@pytest.mark.parametrize("n", [512, 1024, 1500, 2048, 2400, 4096, 6000])
def test_row_sums(n):
    here = plain = 0.0
    for seed in range(8):
        A, x0 = _problem(n, 100 * n + seed)
        here += _first_residual(A, x0) ** 2
        plain += _plain_order(A, x0) ** 2
    assert here <= 1.05 ** 2 * plain, (here / plain) ** 0.5
