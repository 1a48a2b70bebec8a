"""Kernels of a decode step that do two kernels' work: the feed-forward's unit behind the weight-streaming product, and the
short filters that move their state on themselves when every request brings one token."""
import pytest
import torch

from test_muvonex_ops_gpu import dev, step_batch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from nanohybrid_vlm_b200.kernels import ops
    return ops


@pytest.mark.parametrize("unit,mode", [("gelu_tanh_mul", 2), ("relu_squared", 0), ("gelu_tanh", 0)])
@pytest.mark.parametrize("M,inter,K", [(1, 40, 64), (8, 1000, 264), (5, 5632, 2048), (3, 148 * 70, 128)])
def test_unit_behind_the_streaming_product(ops, unit, mode, M, inter, K):
    g = torch.Generator().manual_seed(inter)
    rows = 2 * inter if mode == 2 else inter
    x = dev(torch.randn(M, K, generator=g).to(torch.bfloat16))
    w = dev((torch.randn(rows, K, generator=g) * K ** -0.5).to(torch.bfloat16))
    out = torch.full((M, inter), float("nan"), dtype=torch.bfloat16, device="cuda")
    assert not ops.product_with_unit(out, x, w, unit)             # no copy of the weight
    ops.prepare_streaming(w, mode)
    assert ops.product_with_unit(out, x, w, unit)
    assert not ops.product_with_unit(out, torch.cat([x] * 9)[:9], w, unit)
    y = (x.double() @ w.double().t()).to(torch.bfloat16).double()
    a, u = (y[:, :inter], y[:, inter:]) if mode == 2 else (y, 1.0)
    want = torch.relu(a) ** 2 if unit == "relu_squared" else torch.nn.functional.gelu(a, approximate="tanh") * u
    # the product in bfloat16 may round the other way (2^-8 of values of size 1, doubled by the square), then once more
    torch.testing.assert_close(out.double(), want, rtol=3 * 2 ** -8, atol=2e-3)
    assert ops.slab_error() == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("C,K", [(70, 4), (129, 2), (64, 8), (33, 1)])
def test_filters_on_single_tokens(ops, dtype, C, K):
    """Three requests one token at a time beside an idle entry, then a portion of several: the same as whole portions."""
    g = torch.Generator().manual_seed(C)
    T, slots = 11, [2, 0, 1]
    xs = [torch.randn(T + 3, C, generator=g).to(dtype) for _ in slots]
    w, w2 = (dev((torch.randn(C, K, generator=g) * 0.5).to(dtype)) for _ in range(2))
    bias = dev((torch.randn(C, generator=g) * 0.3).to(dtype))

    def run(cuts):
        states = [torch.full((3, max(K - 1, 1) * C), float("nan"), device="cuda") for _ in range(2)]
        got = [[] for _ in slots]
        for lo, hi in zip([0, *cuts], [*cuts, T + 3]):
            n = hi - lo
            x = torch.cat([x[lo:hi] for x in xs] + [xs[0][:1]])       # behind them an idle entry of one token
            b = step_batch([n] * 3 + [1], [lo] * 3 + [0], slots + [-1])
            y = torch.empty(x.shape, dtype=torch.float32, device="cuda")
            f1, f2 = (torch.empty(x.shape, dtype=dtype, device="cuda") for _ in range(2))
            ops.short_conv_silu(y, dev(x), w, bias, states[0], b)
            ops.causal_filter_add(f1, f2, dev(x), w, w2, states[1], b)
            for r in range(3):
                got[r].append(torch.cat([y[r * n:(r + 1) * n], f1[r * n:(r + 1) * n].float(), f2[r * n:(r + 1) * n].float()], 1))
        return [torch.cat(p) for p in got], states

    single, kept = run(list(range(1, T + 1)))
    whole, want = run([T])
    for a, b in zip(single + (kept if K > 1 else []), whole + (want if K > 1 else [])):
        assert torch.equal(a, b)


def test_as_many_tokens_as_requests_need_not_be_single_tokens(ops):
    """Two tokens, none and one: three tokens of three requests, but no step of single tokens."""
    g = torch.Generator().manual_seed(1)
    C, K, H, d, dv = 64, 4, 2, 16, 16
    x = dev(torch.randn(3, C, generator=g))
    w = dev(torch.randn(C, K, generator=g))
    proj, gates = dev(torch.randn(3, 2 * H * d + H * dv, generator=g)), dev(torch.randn(3, 2 * H, generator=g))
    bias = dev(torch.randn(2 * H, generator=g))
    floats = ops.mlstm_state_floats(H, d, dv)

    def run(steps):
        conv, mem = torch.zeros(3, (K - 1) * C, device="cuda"), torch.zeros(3, floats, device="cuda")
        outs = []
        for rows, news, starts, slots in steps:
            b = step_batch(news, starts, slots)
            y, f = (torch.empty(len(rows), C, device="cuda") for _ in range(2))
            o = torch.empty(len(rows), H * dv, device="cuda")
            ops.causal_filter_add(f, None, x[rows].contiguous(), w, None, conv.clone(), b)
            ops.short_conv_silu(y, x[rows].contiguous(), w, None, conv, b)
            ops.mlstm_scan(o, proj[rows].contiguous(), gates[rows].contiguous(), bias, 15.0, mem, b, H, d, dv)
            outs.append(torch.cat([y, f, o], 1))
        return torch.cat(outs), conv, mem

    for a, b in zip(run([([0, 1, 2], [2, 0, 1], [0, 5, 0], [0, 1, 2])]),
                    run([([0, 1], [2], [0], [0]), ([2], [1], [0], [2])])):
        torch.testing.assert_close(a, b, rtol=1e-5, atol=1e-6)
