"""Which kernel takes a dense solve whose vectors nearly fill the one-exchange kernel's shared memory, at both sides
of the rule; both give the solution (cond 1.5: the true residual stays within a few roundings of 2 tol)."""
import pytest
import torch

import cola_gb300 as cola
from cola_gb300.linalg import cg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,jacobi,kernel", [(16000, False, "k_cg_dense"), (16200, False, "k_cg_fused"),
                                             (16200, True, "k_cg_dense"), (16201, False, "k_cg_dense")])
def test_long_vectors(kernels_of, n, jacobi, kernel):
    # a rank-one update of the identity: eigenvalues 1 and 1 + 0.5
    v = torch.randn(n, generator=torch.Generator("cuda").manual_seed(n), device="cuda")
    v /= v.norm()
    A = 0.5 * v[:, None] * v[None, :]
    A.diagonal().add_(1.0)
    b = torch.randn(n, generator=torch.Generator("cuda").manual_seed(1), device="cuda")
    P = cola.Diagonal(1.0 / A.diagonal()) if jacobi else None
    (x, info), names = kernels_of(lambda: cg(cola.PSD(cola.Dense(A)), b, P=P, tol=1e-5, max_iters=50))
    assert any(kernel in name for name in names), names
    assert info["fused"] and info["iterations"] < 20
    xd, bd, vd = x.double(), b.double(), v.double()
    res = bd - xd - 0.5 * vd * (vd @ xd)
    assert float(res.norm() / bd.norm()) <= 2e-5 + 20 * 1.5 * 2.0 ** -24 * 4
