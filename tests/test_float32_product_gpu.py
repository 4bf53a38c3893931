"""The float32 product on the tensor cores at the edges of its tiles and stages, near the exact sums, and over values that its three
parts do not hold."""

import math

import pytest
import torch

from test_kernels_gpu import ops, rand  # noqa: F401  (ops: a fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(1, 1, 4), (33, 257, 64), (65, 256, 68), (97, 4096, 132), (700, 4100, 260), (1025, 511, 1024), (200, 19000, 192),
                                   (2049, 3000, 128), (12, 300, 4096)])
def test_product_is_near_the_exact_sums(ops, cuda_device, M, N, K):
    x, w = rand((M, K), torch.float32, cuda_device, 1), rand((N, K), torch.float32, cuda_device, 2)
    got, exact = ops.gemm_nt_simt(x, w).double(), x.double() @ w.double().T
    # A stage of 64 values: four cuts of its sum and a rounding of the total, each at most 2^-23 of the sum so far, and the sum's
    # 2-norm grows with the square root; parts left out 2^-24; the output's rounding 2^-24.
    stages = math.ceil(K / 64)
    assert (got - exact).norm() <= exact.norm() * 2.0 ** -23 * (2 + math.sqrt(stages))
    for row in {0, M // 2, M - 1}:
        assert torch.equal(ops.gemm_nt_simt(x[row:row + 1], w).double(), got[row:row + 1])


def test_values_beyond_the_parts(ops, cuda_device):
    """Infinities, NaN, values that round to infinity in bfloat16 and sums near the smallest: as multiply-adds give them."""
    x, w = rand((70, 256), torch.float32, cuda_device, 3), rand((140, 256), torch.float32, cuda_device, 4)
    x[3, 5], x[4, 6], x[5, 7], w[9, 100] = math.inf, math.nan, 3.4e38, -math.inf
    x[6] *= 1e-36
    got, exact = ops.gemm_nt_simt(x, w), x.double() @ w.double().T
    assert torch.equal(got.isnan(), exact.isnan())
    assert torch.equal(got.isinf(), exact.float().isinf()) and torch.equal(got[got.isinf()], exact.float()[got.isinf()])
    rows = [i for i in range(70) if i not in (3, 4, 5)]
    fine = torch.arange(140, device=cuda_device) != 9
    a, b = got[rows][:, fine].double(), exact[rows][:, fine]
    assert ((a - b).norm(dim=1) <= 256 * 2.0 ** -24 * b.norm(dim=1)).all()
