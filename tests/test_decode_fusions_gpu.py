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
