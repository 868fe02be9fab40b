"""The tridiagonal QL: sweeps that overlap the rotations of the one before (two buffers) or wait for them
(one, large m), searches over more than one group of 32, vectors replayed from the recorded rotations or
applied in place, and matrices that split.

An entry passes at most 2 m sweeps, in each through two rotations of error <= 8 u: 32 m u, times |T| for
the eigenvalues and residuals."""
import numpy as np
import pytest
import torch
from scipy.linalg import eigvalsh_tridiagonal

from cola_gb300.linalg.lanczos import tridiag_eigh

pytestmark = pytest.mark.gpu
U = {torch.float32: 2.0 ** -24, torch.float64: 2.0 ** -53}


def _tri(m, dtype, split):
    g = np.random.default_rng(m)
    a, b = g.uniform(1.0, 3.0, (2, m)), g.uniform(0.1, 1.0, (2, max(m - 1, 0)))
    if split:
        b[:, ::7] = 0.0
    return torch.tensor(a).to("cuda", dtype), torch.tensor(b).to("cuda", dtype)


@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("dtype,m,vectors", [(t, m, v) for t in (torch.float32, torch.float64)
                                              for m in (1, 2, 3, 32, 33, 34, 65, 129) for v in (False, True)]
                         + [(torch.float64, 801, True), (torch.float64, 3413, False), (torch.float64, 3414, False)])
def test_tridiag(dtype, m, vectors, split):
    beta, alpha = _tri(m, dtype, split)
    evals, V, status = tridiag_eigh(beta, alpha, want_vectors=vectors)
    assert int(status.abs().max()) == 0
    tol = 32 * m * U[dtype]
    for s in range(2):
        a, b = beta[s].double().cpu().numpy(), alpha[s].double().cpu().numpy()
        want = eigvalsh_tridiagonal(a, b) if m > 1 else a
        assert np.abs(evals[s].double().cpu().numpy() - want).max() <= 5 * tol
        W = V[s].double()
        if vectors:
            T = torch.diag(beta[s].double())
            T = T + torch.diag(alpha[s].double(), 1) + torch.diag(alpha[s].double(), -1)
            assert float((W.T @ W - torch.eye(m, device="cuda", dtype=torch.float64)).abs().max()) <= 2 * tol
            assert float((T @ W - W * evals[s].double()).norm(dim=0).max()) <= 10 * tol
        else:
            assert abs(float((W * W).sum()) - 1.0) <= 2 * tol
            assert abs(float((W * W * evals[s].double()).sum()) - a[0]) <= 10 * tol
