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


def both(ops, x, w):
    out, simt = (torch.full((x.shape[0], w.shape[0]), float("nan"), device="cuda") for _ in range(2))
    assert ops._f32_on_tensor_cores(x, w)
    ops.linear(out, x, w)
    ops.linear_simt(simt, x, w)
    ops.raise_wait_errors()
    return out, simt


def same(a, b):
    """The same values: infinities with their sign, and what is no number in the same places."""
    return torch.equal(a.isnan(), b.isnan()) and torch.equal(a[~a.isnan()], b[~b.isnan()])


# one run of K and four; tiles of 32 and of 128 rows
SHAPES = pytest.mark.parametrize("M,N,K", [(20, 6400, 516), (140, 6400, 516), (20, 700, 1092), (140, 700, 1092)])


@SHAPES
@pytest.mark.parametrize("scale", [1e-33, 1e-36, 1e-41])
def test_rows_below_what_three_bfloat16_hold(ops, M, N, K, scale):
    """Rows of either operand whose last bits are below bfloat16's smallest number, down to fp32's own last numbers: what fp32
    multiply-adds give; the rows beside them keep their bits."""
    x, w = operands(M, N, K)
    clean, _ = both(ops, x, w)
    x2, w2 = x.clone(), w.clone()
    x2[[3, M - 1]] *= scale
    w2[[0, N - 1]] *= scale
    out, simt = both(ops, x2, w2)
    assert torch.equal(out[[3, M - 1]], simt[[3, M - 1]]) and torch.equal(out[:, [0, N - 1]], simt[:, [0, N - 1]])
    rest = [i for i in range(M) if i not in (3, M - 1)]
    assert torch.equal(out[rest][:, 1:-1], clean[rest][:, 1:-1])
    x2[3], x2[M - 1] = 0, x[M - 1]                          # a row of zeros; a row with one ordinary value
    x2[M - 1, 1:] *= scale
    out, simt = both(ops, x2, w2)
    assert (out[3] == 0).all() and torch.equal(out[rest[:3]][:, 1:-1], clean[rest[:3]][:, 1:-1])
    # one product, of which the parts leave out 2^-24, and what is 2^-30 of it
    torch.testing.assert_close(out[M - 1, 1:-1], (x2[M - 1, 0] * w[:, 0])[1:-1], rtol=2 ** -22, atol=0)


@SHAPES
def test_infinities_and_sums_beyond_the_range(ops, M, N, K):
    x, w = operands(M, N, K)
    clean, _ = both(ops, x, w)
    inf = float("inf")
    for places in ([(0, inf)], [(K - 1, -inf)], [(1, inf), (K - 2, -inf)], [(5, float("nan"))]):
        x2, w2 = x.clone(), w.clone()
        for k, v in places:
            x2[M - 1, k], w2[N - 1, k] = v, v
        out, simt = both(ops, x2, w2)
        assert same(out[M - 1], simt[M - 1]) and same(out[:, N - 1], simt[:, N - 1])
        assert torch.equal(out[:-1, :-1], clean[:-1, :-1])
    x2 = x.clone()
    x2[M - 1] *= 1e37                                       # some of the sums are beyond the range, and parts of others on the way
    out, simt = both(ops, x2, w)
    over = ~out[M - 1].isfinite()
    assert over.any() and not over.all() and same(out[M - 1][over], simt[M - 1][over])
    assert out[M - 1][simt[M - 1].isfinite()].isfinite().all() and torch.equal(out[:-1], clean[:-1])


@SHAPES
def test_values_above_the_largest_bfloat16(ops, M, N, K):
    x, w = operands(M, N, K)
    x[M - 1] = 0
    x[M - 1, 7], x[M - 1, K - 1] = 3.4e38, -torch.finfo(torch.float32).max
    w *= 0.01
    out, _ = both(ops, x, w)
    want = x[M - 1].to(F64) @ w.to(F64).T
    size = x[M - 1].abs().to(F64) @ w.abs().to(F64).T
    assert ((out[M - 1].to(F64) - want).abs() <= 2 ** -22 * size).all()


@SHAPES
def test_sums_near_the_smallest_number(ops, M, N, K):
    """Sums that fp32 holds with fewer bits, by operands of ordinary size: what multiply-adds give."""
    x, w = operands(M, N, K)
    out, simt = both(ops, x * 1e-20, w * 1e-20)
    assert simt.abs().max() < 1e-37 and torch.equal(out, simt)
    x[1] *= 1e-20                                           # beside others: the row by itself
    out, simt = both(ops, x, w * 1e-17)
    want = x.to(F64) @ (w * 1e-17).to(F64).T
    off, off_simt = ((o.to(F64) - want)[1].norm() for o in (out, simt))
    assert off <= off_simt


def test_operands_of_one_sign(ops):
    """The tensor cores cut sums off instead of rounding them, always to one side: still no further off than multiply-adds."""
    g = torch.Generator().manual_seed(1)
    for K in (512, 4096):
        x, w = torch.rand(40, K, generator=g).cuda(), torch.rand(516, K, generator=g).cuda()
        want = x.to(F64) @ w.to(F64).T
        off, off_simt = ((o.to(F64) - want).norm() for o in both(ops, x, w))
        assert off <= off_simt
