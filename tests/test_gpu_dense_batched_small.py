"""The uneven dense batch at sizes where its partition can go wrong: one-row systems, rows of a few quads,
row pairs and their limit of 512 entries, every row alignment, more systems than a warp scans at once and
systems that stop at different steps.  Each against a dense FP64 solve.

Tolerance: K = 1.6 I + E with |E| < 1 gives cond <= 5; FP32 CG stops at a recursive residual of 2e-6 and
adds at most s n^(1/2) u for s <= 60 steps, so |x - x*| / |x*| <= 5 (2e-6 + 60 sqrt(600) 2^-24) = 4.5e-4."""
import pytest
import torch

from cola_gb300.linalg import solve_dense_batched

pytestmark = pytest.mark.gpu


def _batch(sizes, seed):
    g = torch.Generator("cuda").manual_seed(seed)
    mats, rhs = [], []
    for n in sizes:
        M = torch.randn(n, n, generator=g, device="cuda", dtype=torch.float64) / (2 * n ** 0.5)
        E = 0.5 * (M + M.T)
        E = E / max(1.0, 1.01 * float(torch.linalg.matrix_norm(E, 2)))
        mats.append((E + 1.6 * torch.eye(n, device="cuda", dtype=torch.float64)).float())
        rhs.append(torch.randn(n, generator=g, device="cuda"))
    return mats, rhs


@pytest.mark.parametrize("sizes", [[1], [2, 1, 3], [5, 511, 512, 513, 514, 515], list(range(1, 72)), [600, 33, 257, 1, 130, 599]])
def test_small_batches(sizes):
    mats, rhs = _batch(sizes, len(sizes))
    xs, iters, status = solve_dense_batched(mats, rhs, tol=1e-6, max_iters=200)
    assert bool((status == 1).all()) and int(iters.max()) <= 60
    for A, b, x in zip(mats, rhs, xs):
        e = torch.linalg.solve(A.double(), b.double())
        assert float((x.double() - e).norm() / e.norm()) <= 4.5e-4
