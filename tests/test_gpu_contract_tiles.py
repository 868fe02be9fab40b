"""The contraction's tiles of many sums a thread, in every staging form: asynchronous copies (FP32, and BF16 rows beside
FP32 columns), registers, and columns of few entries; M, K and N at the edges of the tiles, columns that straddle
a Kronecker block, whole and ragged quads of the output.

Tolerance: a K-term sum in any order is within K u sum |a x| of the exact one, plus one rounding of the result.
Sums in the plain order of k are the same to the bit in every tile, so a product's columns may not depend on how
many others are formed with them."""
import pytest
import torch

import cola_gb300 as cola

pytestmark = pytest.mark.gpu
U = 2.0 ** -24


def _rand(*shape, dtype, seed=0):
    return torch.randn(*shape, generator=torch.Generator("cuda").manual_seed(seed), device="cuda").to(dtype)


# 128 x 16; 48 and 64 x 128; 64 x 64 in slices of 16 and of 32; long sums through registers
SHAPES = [(39000, 16, 16), (38945, 17, 9), (40001, 33, 5), (96, 48, 20480), (48, 47, 36868), (144, 63, 13001), (16, 16, 50000),
          (64, 64, 36864), (128, 200, 18004), (1000, 100, 1000), (1001, 127, 1003), (1000, 256, 1000), (999, 129, 1001),
          (1001, 700, 1003), (1000, 700, 1000), (641, 1030, 61)]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("M,K,N", SHAPES)
def test_products(M, K, N, dtype):
    A, X = _rand(M, K, dtype=dtype, seed=1), _rand(K, N, dtype=torch.float32, seed=2)
    Y = cola.ops.Dense(A) @ X
    E, scale = A.double() @ X.double(), A.double().abs() @ X.double().abs()
    assert bool(((Y.double() - E).abs() <= (K + 1) * U * scale).all())
    if K <= 256:  # the first columns alone: another tile, the same bits
        few = cola.ops.Dense(A) @ X[:, :5].contiguous()
        assert torch.equal(few, Y[:, :5])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("dims,k", [((48, 48, 48), 9), ((96, 300), 5), ((300, 96), 3), ((64, 640), 1), ((640, 64), 2),
                                    ((130, 500), 2), ((500, 130), 3), ((63, 65, 20), 5)])
def test_kronecker(dims, k, dtype):
    Ks = [_rand(m, m, dtype=dtype, seed=i) for i, m in enumerate(dims)]
    n = 1
    for m in dims:
        n *= m
    X = _rand(n, k, dtype=torch.float32, seed=9)
    Y = cola.ops.Kronecker(*[cola.ops.Dense(K) for K in Ks], precision="fp32") @ X
    E, S = X.double().reshape(*dims, k), X.double().abs().reshape(*dims, k)
    for i, K in enumerate(Ks):
        E = torch.movedim(torch.tensordot(K.double(), E, dims=([1], [i])), 0, i)
        S = torch.movedim(torch.tensordot(K.double().abs(), S, dims=([1], [i])), 0, i)
    tol = sum(m + 1 for m in dims) * U * S.reshape(n, k) * 1.01  # first order in u
    assert bool(((Y.double() - E.reshape(n, k)).abs() <= tol).all())
    one = cola.ops.Kronecker(*[cola.ops.Dense(K) for K in Ks], precision="fp32") @ X[:, :1].contiguous()
    if max(dims) <= 256:
        assert torch.equal(one, Y[:, :1])


@pytest.mark.parametrize("beta", [0.0, -0.5])
def test_accumulation(beta):
    """Y = A X + beta Y as the sum of two operators, at a tile that stores whole quads and one that does not."""
    for N in (1000, 1001):
        A, B = _rand(1000, 200, dtype=torch.float32, seed=1), _rand(1000, 200, dtype=torch.float32, seed=3)
        X = _rand(200, N, dtype=torch.float32, seed=2)
        Y = (beta * cola.ops.Dense(B) + cola.ops.Dense(A)) @ X
        E = A.double() @ X.double() + beta * (B.double() @ X.double())
        S = A.double().abs() @ X.double().abs() + abs(beta) * (B.double().abs() @ X.double().abs())
        assert bool(((Y.double() - E).abs() <= 203 * U * S).all())
