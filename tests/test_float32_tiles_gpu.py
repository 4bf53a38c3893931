"""The 32-bit kernels that work in register tiles, alone: the product at the edges of its tiles and of its slices of k."""

import math

import pytest
import torch

from test_kernels_gpu import ops, rand  # noqa: F401  (ops: a fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(1, 32, 4), (31, 33, 64), (33, 100, 60), (64, 128, 16), (700, 1024, 132), (640, 1000, 1028),
                                   (1281, 515, 68)])
def test_product_at_tile_edges(ops, cuda_device, M, N, K):
    x, w = rand((M, K), torch.float32, cuda_device, 1), rand((N, K), torch.float32, cuda_device, 2)
    got = ops.gemm_nt_simt(x, w)
    # A sum of K products: every partial sum is rounded, at most K of them of magnitude up to sqrt(K) times a few.
    assert (got.double() - x.double() @ w.double().T).abs().max() <= 6 * 2.0 ** -24 * math.sqrt(K) * math.sqrt(K)
    # A row's sums are the same on either tile size and in a batch of any size.
    assert torch.equal(ops.gemm_nt_simt(x[M - 1:], w), got[M - 1:])
    # Rows that lie apart, in and out; what lies between them stays.
    wide = torch.full((M, N + 3), 7.0, device=cuda_device)
    ops.gemm_nt_simt(rand((M, K), torch.float32, cuda_device, 1).repeat(1, 2)[:, :K], w, out=wide[:, :N])
    assert torch.equal(wide[:, :N], got) and bool((wide[:, N:] == 7.0).all())
