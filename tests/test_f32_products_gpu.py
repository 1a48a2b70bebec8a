"""Float32 products on the tensor cores (operands as three bfloat16, csrc/gemm_f32_tcgen05.cu): at the edges of tiles, stages and
runs of K, against 64 bits and the CUDA-core product; the same bits for any number of rows; values that are no number."""
import pytest
import torch

pytestmark = pytest.mark.gpu
F64 = torch.float64


@pytest.fixture(scope="module")
def ops():
    from nanohybrid_vlm_b200.kernels import ops as module
    return module


def operands(M, N, K, seed=0, scale=1.0):
    g = torch.Generator().manual_seed(seed + K)
    return (torch.randn(M, K, generator=g) * scale).cuda(), torch.randn(N, K, generator=g).cuda()


# K: one run with an odd last stage, two and four runs, a last run shorter than the others; N: off the tile, above the sizes
# that are cut into runs
@pytest.mark.parametrize("N,K", [(512, 512), (513, 516), (640, 580), (1024, 1032), (1100, 2048), (700, 1092), (6400, 516), (7001, 512)])
def test_products(ops, N, K):
    x, w = operands(300, N, K)
    want = x.to(F64) @ w.to(F64).T
    whole = torch.full((300, N), float("nan"), device="cuda")
    assert ops._f32_on_tensor_cores(x, w)
    ops.linear(whole, x, w)
    simt = torch.empty_like(whole)
    ops.linear_simt(simt, x, w)
    off, off_simt = ((o.to(F64) - want).norm() / want.norm() for o in (whole, simt))
    assert off <= off_simt, (off, off_simt)
    # 64 columns are added up at a time with four sums cut off at 2^-23, then K / 64 times rounded to 2^-24: all of one sign
    # and each as large as the largest sum of K unit products (5 K^1/2) they make this
    assert (whole.to(F64) - want).abs().max().item() <= (4 + K / 128) * 2 ** -23 * 5 * K ** 0.5
    for M in (1, 2, 31, 32, 33, 127, 128, 129):             # other tiles, the same bits
        out = torch.full((M + 1, N), float("nan"), device="cuda")
        ops.linear(out[:M], x[300 - M:], w)
        assert torch.equal(out[:M], whole[300 - M:]) and out[M].isnan().all()
    ops.raise_wait_errors()


def test_large_and_small_values(ops):
    for scale in (1e30, 1e-30):
        x, w = operands(40, 516, 512, scale=scale)
        out = torch.empty(40, 516, device="cuda")
        ops.linear(out, x, w)
        want = x.to(F64) @ w.to(F64).T
        assert ((out.to(F64) - want).norm() / want.norm()).item() < 3e-7


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), float("-inf")])
def test_a_value_that_is_no_number_stays_in_its_row_and_column(ops, bad):
    x, w = operands(70, 600, 516)
    clean, got = torch.empty(70, 600, device="cuda"), torch.empty(70, 600, device="cuda")
    ops.linear(clean, x, w)
    x2, w2 = x.clone(), w.clone()
    x2[37, 515] = bad
    w2[129, 3] = bad
    ops.linear(got, x2, w2)
    rows, cols = [i for i in range(70) if i != 37], [i for i in range(600) if i != 129]
    assert torch.equal(got[rows][:, cols], clean[rows][:, cols])
    assert not got[37].isfinite().any() and not got[:, 129].isfinite().any()


def test_what_the_tensor_cores_do_not_take_goes_to_the_cuda_cores(ops):
    x, w = operands(9, 600, 516)
    wide = torch.randn(9, 519, device="cuda")
    wide[:, :516] = x
    small = torch.randn(200, 516, device="cuda")
    for a, b in ((wide[:, :516], w), (x, small), (x[:, 1:].contiguous(), w[:, 1:].contiguous()), (x[:, :508].contiguous(), w[:, :508].contiguous())):
        assert not ops._f32_on_tensor_cores(a, b)
        out, simt = (torch.empty(9, b.shape[0], device="cuda") for _ in range(2))
        ops.linear(out, a, b)
        ops.linear_simt(simt, a, b)
        assert torch.equal(out, simt)
