"""The CUDA-core product at the edges of its tiles, and where sizes or addresses send it another way (operands that cannot
be copied 16 bytes at a time), against a 64-bit reference and against each other."""
import pytest
import torch

pytestmark = pytest.mark.gpu

F64 = torch.float64


@pytest.fixture(scope="module")
def ops():
    from nanohybrid_vlm_b200.kernels import ops
    return ops


# the tiles are 16 x 32, 32 x 64 and 64 x 64 outputs and 32 columns of k; the largest tile serves the widest sizes here
@pytest.mark.parametrize("M,N,K", [(1, 32, 32), (16, 33, 36), (17, 64, 28), (31, 65, 64), (33, 4096, 100), (64, 6144, 32),
                                   (370, 4100, 68), (370, 1024, 2048)])
def test_product_at_tile_edges_and_with_unaligned_operands(ops, M, N, K):
    g = torch.Generator().manual_seed(M + N)
    wide = torch.randn(M, K + 5, generator=g).cuda()
    w = torch.randn(N, K, generator=g).cuda()
    ref = wide[:, :K].to(F64) @ w.to(F64).t()
    plain, moved = torch.empty(M, N, device="cuda"), torch.empty(M, N, device="cuda")
    ops.linear_simt(plain, wide[:, :K].contiguous(), w)
    # 32-bit sums of K products of unit variance: K / 2 additions to each of two sums
    bound = 2 ** -23 * K ** 0.5 * (K / 2 + 2)
    assert (plain.to(F64) - ref).abs().max().item() < bound
    ops.linear_simt(moved, wide[:, :K], w)               # rows K + 5 apart: no 16-byte copies
    assert torch.equal(plain, moved)
