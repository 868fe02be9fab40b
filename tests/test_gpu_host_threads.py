"""Solves of different sizes from two host threads on two streams: what a launch may use depends on its own
call alone, so every call completes, with the bits it gives alone."""
import threading
import time

import pytest
import torch

import cola_gb300 as cola
from cola_gb300.linalg import BatchedCSR, cg, solve_batched
from cola_gb300.linalg.lanczos import run_lanczos

pytestmark = pytest.mark.gpu


def _dense(n):  # the grid form of the fused dense CG, rows resident
    M = torch.randn(n, n, generator=torch.Generator("cuda").manual_seed(n), device="cuda") / (2.0 * n ** 0.5)
    op = cola.PSD(cola.Dense(0.5 * (M + M.T) + 2.0 * torch.eye(n, device="cuda")))
    b = torch.ones(n, device="cuda")
    return lambda: cg(op, b, tol=0.0, max_iters=10)[0]


def _step_tail(k):  # the generic loop's step as one cluster
    F = cola.Dense(torch.diag(torch.linspace(1.0, 2.0, 16, device="cuda")))
    op = cola.PSD(cola.Kronecker(F, F))
    b = torch.ones(256, k, device="cuda")
    return lambda: cg(op, b, tol=0.0, max_iters=10)[0]


def _block(m, k=16):  # many right-hand sides of one matrix: the block schedule
    n = m * m
    p = torch.arange(n, device="cuda")
    cols = torch.stack([p - m, p - 1, p, p + 1, p + m], 1)
    ok = torch.stack([p >= m, p % m > 0, p >= 0, p % m < m - 1, p < n - m], 1)
    vals = torch.tensor([-1.0, -1.0, 5.0, -1.0, -1.0], device="cuda").expand(n, 5)[ok]
    indptr = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
    indptr[1:] = torch.cumsum(ok.sum(1), 0)
    fam = BatchedCSR(indptr, cols[ok].to(torch.int32), vals[None].contiguous(), shared=True)
    B = torch.ones(k, n, dtype=torch.float64, device="cuda")
    return lambda: solve_batched(fam, B, precond="jacobi", tol=1e-6)[0]


def _lanczos(n):  # a run of the vector per CTA in shared memory
    op = cola.SelfAdjoint(cola.Diagonal(torch.linspace(1.0, 2.0, n, device="cuda")))
    v = torch.ones(n, 1, device="cuda")
    return lambda: run_lanczos(op, v, 12, 0.0).basis


@pytest.mark.parametrize("make,sizes", [(_dense, (2000, 800)), (_step_tail, (512, 1)), (_block, (200, 20)),
                                        (_lanczos, (2000000, 40000))])
def test_different_sizes_on_two_threads(make, sizes):
    calls = [make(s) for s in sizes]
    alone = [f() for f in calls]
    torch.cuda.synchronize()
    errors, stop, end = [], threading.Event(), time.monotonic() + 3.0

    def work(f, expect):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                while not stop.is_set() and time.monotonic() < end:
                    if not torch.equal(f(), expect):
                        raise AssertionError("another result than alone")
        except Exception as e:  # noqa: BLE001 - reported by the test below
            errors.append(repr(e))
            stop.set()

    threads = [threading.Thread(target=work, args=a) for a in zip(calls, alone)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
