"""Dense and Kronecker products in the contraction kernel against FP64 torch, at tile edges, odd sizes,
split k ranges, the columns that straddle a Kronecker block, and every storage type.

Tolerance: a K-term sum in any order is within K * u * sum |a x| of the exact one (u the compute type's
unit roundoff); plus one rounding of the result."""
import pytest
import torch

import cola_gb300 as cola

pytestmark = pytest.mark.gpu
U = {torch.float32: 2.0 ** -24, torch.float64: 2.0 ** -53, torch.bfloat16: 2.0 ** -24}


def _rand(*shape, dtype, seed=0):
    return torch.randn(*shape, generator=torch.Generator("cuda").manual_seed(seed), device="cuda",
                       dtype=torch.float64).to(dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, torch.bfloat16])
@pytest.mark.parametrize("M,K,N", [(1, 1, 5), (3, 5, 7), (32, 64, 8), (33, 65, 9), (48, 48, 4096), (64, 96, 130),
                                   (47, 33, 70), (65, 515, 33), (130, 1500, 16), (1000, 1024, 64), (1500, 700, 17),
                                   (2000, 300, 320)])
def test_dense_products(M, K, N, dtype):
    A = _rand(M, K, dtype=dtype, seed=1)
    X = _rand(K, N, dtype=torch.float64 if dtype == torch.float64 else torch.float32, seed=2)
    Y = cola.ops.Dense(A) @ X
    E, scale = A.double() @ X.double(), A.double().abs() @ X.double().abs()
    slack = 2.0 if dtype == torch.float64 else 1.0  # the FP64 reference itself rounds
    assert bool(((Y.double() - E).abs() <= slack * (K + 1) * U[dtype] * scale).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("dims,k", [((7, 9), 1), ((7, 9), 2), ((33, 17, 5), 3), ((48, 48, 6), 5), ((96, 80), 8),
                                    ((512, 3), 1), ((3, 300), 4), ((64, 64), 31)])
def test_kronecker_products(dims, k, dtype):
    Ks = [_rand(m, m, dtype=dtype, seed=i) for i, m in enumerate(dims)]
    n = 1
    for m in dims:
        n *= m
    X = _rand(n, k, dtype=dtype, seed=9)
    Y = cola.ops.Kronecker(*[cola.ops.Dense(K) for K in Ks], precision="fp32") @ X
    E, S = X.double().reshape(*dims, k), X.double().abs().reshape(*dims, k)
    for i, K in enumerate(Ks):
        E = torch.movedim(torch.tensordot(K.double(), E, dims=([1], [i])), 0, i)
        S = torch.movedim(torch.tensordot(K.double().abs(), S, dims=([1], [i])), 0, i)
    slack = 2.0 if dtype == torch.float64 else 1.0
    tol = slack * sum(m + 1 for m in dims) * U[dtype] * S.reshape(n, k) * 1.01  # first order in u
    assert bool(((Y.double() - E.reshape(n, k)).abs() <= tol).all())


def test_row_stride_blockdiag_and_empty():
    B = _rand(40, 30, dtype=torch.float32)[:, :29]  # rows 30 floats apart, 29 used
    X = _rand(87, 11, dtype=torch.float32, seed=3)
    Y = cola.ops.BlockDiag(cola.ops.Dense(B), multiplicities=[3]) @ X
    E = torch.cat([B.double() @ X[29 * i: 29 * (i + 1)].double() for i in range(3)])
    S = torch.cat([B.double().abs() @ X[29 * i: 29 * (i + 1)].double().abs() for i in range(3)])
    assert bool(((Y.double() - E).abs() <= 30 * U[torch.float32] * S).all())
    Z = cola.ops.Dense(torch.zeros(5, 0, device="cuda")) @ torch.zeros(0, 7, device="cuda")
    assert Z.shape == (5, 7) and float(Z.abs().max()) == 0.0
