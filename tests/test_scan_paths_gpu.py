"""The recurrent kernels' other ways through a step (single tokens of the mLSTM streamed through; prompts 64 tokens at a
time), against plain recurrences in 64 bits: portions that end at, before and behind a chunk, single tokens beside them,
states handed from one way to the other, heads of less than a kernel's width, columns that are no multiple of 16."""
import pytest
import torch

from test_muvonex_ops_gpu import F64, dev, portions_of, step_batch
from test_nomudra_ops_gpu import mlstm_inputs, plain_scan

pytestmark = pytest.mark.gpu

SLOTS = [1, 3, 0, 2]


@pytest.fixture(scope="module")
def ops():
    from nanohybrid_vlm_b200.kernels import ops
    return ops


def walk(step, width, state, lengths, cuts):
    """All requests through ``step(out, [(request, start, tokens)], batch)``, portion by portion."""
    got = [torch.zeros(n, width) for n in lengths]
    for who, starts, news in portions_of(lengths, cuts):
        o = torch.full((sum(news), width), float("nan"), dtype=torch.float32, device="cuda")
        step(o, [(r, s, n) for r, s, n in zip(who, starts, news)], step_batch(news, starts, [SLOTS[r] for r in who]))
        at = 0
        for r, s, n in zip(who, starts, news):
            got[r][s:s + n] = o[at:at + n].cpu()
            at += n
    kept = state.clone()
    for n in (1, lengths[0]):
        o = torch.full((n, width), float("nan"), dtype=torch.float32, device="cuda")
        step(o, [(0, 0, n)], step_batch([n], [0], [-1]))               # no slot: zeros, and no state moves
        assert (o == 0).all() and torch.equal(state.nan_to_num(7.0), kept.nan_to_num(7.0))
    return got


def rows(parts, which):
    return dev(torch.cat([which[r][s:s + n] for r, s, n in parts]))


def cancellation(proj, gates, bias, H, d):
    """Per token and head of the mLSTM: the sum of the sizes of the normaliser's terms over the normaliser."""
    T, x, raw = proj.shape[0], proj.to(F64), 15.0 * torch.tanh((gates.to(F64) + bias.to(F64)) / 15.0)
    q, k = (x[:, a * H * d:(a + 1) * H * d].view(T, H, d).transpose(0, 1) for a in (0, 1))
    i, f = raw[:, :H].t(), torch.nn.functional.logsigmoid(raw[:, H:]).t().cumsum(-1)
    size = i[:, None, :] + f[:, :, None] - f[:, None, :]
    size = size.masked_fill(torch.ones(T, T, dtype=torch.bool).triu(1), float("-inf"))
    m = torch.maximum(size.amax(-1), f)                     # the running maximum starts at 0
    terms = torch.exp(size - m[..., None]) * (q @ k.transpose(1, 2)) * d ** -0.5
    return (terms.abs().sum(-1) / torch.maximum(terms.sum(-1).abs(), torch.exp(-m))).t()


def check_mlstm(ops, dtype, H, d, dv, spread, lengths, cuts):
    g = torch.Generator().manual_seed(d)
    ins = [mlstm_inputs(g, n, H, d, dv, dtype, spread) for n in lengths]
    ins = [(p[:, :2 * H * d + H * dv].contiguous(), gt) for p, gt in ins]
    bias = torch.cat((torch.randn(H, generator=g), 2 + torch.randn(H, generator=g)))
    state = torch.full((4, -(-ops.mlstm_state_floats(H, d, dv) // 4) * 4), float("nan"), device="cuda")

    def step(o, parts, batch):
        ops.mlstm_scan(o, rows(parts, [i[0] for i in ins]), rows(parts, [i[1] for i in ins]), dev(bias), 15.0, state, batch,
                       H, d, dv)

    for got, (proj, gates) in zip(walk(step, H * dv, state, lengths, cuts), ins):
        want = plain_scan(proj, gates, bias, 15.0, H, d, dv)
        # the normaliser is a sum that may cancel: its relative error is that of 32-bit sums of a few hundred terms
        # (4e-6, some 64 units of 2^-24) times the terms' sizes over what is left of them, and so is the output's
        loss = cancellation(proj, gates, bias, H, d).repeat_interleave(dv, 1)
        assert ((got.to(F64) - want).abs() <= 2e-5 + (2e-4 + 4e-6 * loss) * want.abs()).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,d,dv,spread", [(2, 128, 256, 4.0), (3, 64, 20, 8.0), (1, 100, 36, 1.0), (2, 4, 16, 3.0), (1, 132, 16, 2.0),
                                           (1, 512, 20, 2.0), (1, 260, 7, 2.0)])
def test_mlstm_single_tokens(ops, dtype, H, d, dv, spread):
    """From the first token on, one at a time, three requests side by side; two tokens at once in between."""
    lengths = [9, 7, 3]
    check_mlstm(ops, dtype, H, d, dv, spread, lengths, [[1, 2, 3, 5, 6, 7, 8], [1, 2, 3, 4, 5, 6], [1, 2]])
