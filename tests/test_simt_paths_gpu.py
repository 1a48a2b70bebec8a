"""The CUDA-core product and attention at the edges of their tiles, and where sizes or addresses send them another way
(what cannot be read 16 bytes at a time), against a 64-bit reference and each other."""
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


@pytest.mark.parametrize("planes", [2, 1])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nq,nkv,d,dv,window", [(2, 1, 128, 128, 0), (4, 2, 256, 132, 0), (8, 1, 36, 20, 40), (10, 1, 64, 64, 0)])
def test_attention_in_groups_of_four_agrees_with_the_general_kernel(ops, dtype, nq, nkv, d, dv, window, planes):
    """Requests whose portions leave 1, 2, 3, 8 and 9 pairs to a warp and end at, before and behind a chunk of 32 keys."""
    g = torch.Generator().manual_seed(d)
    lens, news = [1, 31, 32, 33, 96, 130, 7], [1, 2, 32, 5, 1, 40, 7]
    page, n_pages = 8, 60
    pages = torch.full((n_pages, planes, nkv, page, max(d, dv)), float("nan"))
    order, bt = torch.randperm(n_pages, generator=g).tolist(), torch.full((len(lens), 17), -1, dtype=torch.int32)
    for r, n in enumerate(lens):
        for j in range(-(-n // page)):
            bt[r, j] = order.pop()
            pages[bt[r, j], :, :, :min(page, n - j * page)] = torch.randn(planes, nkv, min(page, n - j * page), max(d, dv),
                                                                          generator=g)
    pages = pages.to(dtype).cuda()
    T = sum(news)
    wide = torch.randn(T, nq * d + 1, generator=g).to(dtype).cuda()
    sinks = torch.randn(nq, generator=g).cuda()
    cu = torch.tensor([0] + torch.tensor(news).cumsum(0).tolist(), dtype=torch.int32).cuda()
    kv = torch.tensor(lens, dtype=torch.int32).cuda()
    outs = []
    for q in (wide[:, :nq * d].contiguous(), wide[:, :nq * d]):          # the second: rows an odd number of elements apart
        out = torch.full((T, nq * dv), float("nan"), dtype=dtype, device="cuda")
        ops.attention_sink_simt(out, q, pages, bt.cuda(), cu, kv, len(lens), T, nq, nkv, d, dv, d ** -0.5, sinks, window=window)
        outs.append(out.float())
    # the same chunks in the same order; sums inside a score in another order, bf16 results may round the other way
    tol = dict(rtol=2e-5, atol=2e-5) if dtype == torch.float32 else dict(rtol=2 ** -7, atol=1e-3)
    torch.testing.assert_close(outs[0], outs[1], **tol)
