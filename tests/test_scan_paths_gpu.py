"""The recurrent kernels' other ways through a step (single tokens of the mLSTM streamed through; prompts 32 tokens at a
time), against plain recurrences in 64 bits: portions that end at, before and behind a chunk, single tokens beside them,
states handed from one way to the other, heads of less than a kernel's width, columns that are no multiple of 16."""
import pytest
import torch

from test_muvonex_ops_gpu import F64, delta_inputs, dev, plain_delta, plain_ssd, portions_of, step_batch
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
        # Per token and head, relative to the row: the logarithms of the gates, up to 15, are known to four units of tanh's
        # last place (15 * 4 * 2^-24 = 4e-6), those of some hundred tokens add up (16 times that as a random walk, 6e-5),
        # and numerator and normaliser are sums that may cancel.  (The scan by tokens is off as far at the same tokens.)
        loss = cancellation(proj, gates, bias, H, d)
        off = (got.to(F64) - want).view(-1, H, dv).norm(dim=-1) / want.view(-1, H, dv).norm(dim=-1)
        assert (off <= 6e-5 * (1 + loss)).all(), (off / (1 + loss)).max()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,d,dv,spread", [(2, 128, 256, 4.0), (3, 64, 20, 8.0), (1, 100, 36, 1.0), (2, 4, 16, 3.0), (1, 132, 16, 2.0),
                                           (1, 512, 20, 2.0), (1, 260, 7, 2.0)])
def test_mlstm_single_tokens(ops, dtype, H, d, dv, spread):
    """From the first token on, one at a time, three requests side by side; two tokens at once in between."""
    lengths = [9, 7, 3]
    check_mlstm(ops, dtype, H, d, dv, spread, lengths, [[1, 2, 3, 5, 6, 7, 8], [1, 2, 3, 4, 5, 6], [1, 2]])


@pytest.mark.parametrize("pad", [0, 4])
@pytest.mark.parametrize("H,d,dv,spread", [(2, 128, 256, 4.0), (4, 100, 36, 1.0), (4, 64, 64, 8.0), (4, 512, 20, 2.0), (1, 132, 16, 2.0)])
def test_mlstm_in_a_fixed_order_has_the_same_bits_for_every_cutting(ops, H, d, dv, spread, pad):
    """Whole prompts, single tokens side by side, single tokens beside a portion; slots as the engine makes them, and slots
    that all start on 16 bytes."""
    g = torch.Generator().manual_seed(d)
    lengths = [70, 41, 9]
    ins = [mlstm_inputs(g, n, H, d, dv, torch.float32, spread) for n in lengths]
    bias = dev(torch.cat((torch.randn(H, generator=g), 2 + torch.randn(H, generator=g))))
    floats = ops.mlstm_state_floats(H, d, dv)
    seen = []
    for cuts in ([[], [], []], [list(range(1, n)) for n in lengths], [[1, 2, 40, 41, 42], [1, 2, 3, 4, 40], [1, 2, 3, 4]]):
        state = torch.full((4, -(-floats // 4) * 4 if pad else floats), float("nan"), device="cuda")

        def step(o, parts, batch):
            ops.mlstm_scan(o, rows(parts, [i[0] for i in ins]), rows(parts, [i[1] for i in ins]), bias, 15.0, state, batch,
                           H, d, dv, fixed_order=True)

        got = walk(step, H * dv, state, lengths, cuts)
        seen.append(got + [state[SLOTS[r], :floats].cpu() for r in range(3)])
    for other in seen[1:]:
        for a, b in zip(seen[0], other):
            assert torch.equal(a, b)


# ---------------------------------------------------------------- prompts, 32 tokens at a time
LENGTHS = [200, 129, 64, 70]
# per step: 65, 64, 31, 1 tokens; then 1, 1, 33, 68; then 133, 64, -, 1; then a single token
CUTS = [[65, 66, 199], [64, 65], [31], [1, 69]]
# 32-bit sums of up to 128 products per element and chunk, states over 200 tokens; the scans by tokens are held to the same
TOL = dict(rtol=3e-5, atol=3e-5)


@pytest.fixture
def chunks(ops):
    """The scans by chunks at every step of 16 tokens a request, whatever the rule would choose."""
    ops.CHUNK_SCAN_TOKENS = 16
    yield
    ops.CHUNK_SCAN_TOKENS = 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("G,H,d,dv", [(2, 4, 128, 128), (1, 5, 64, 20), (3, 3, 100, 36), (1, 2, 16, 16), (2, 2, 4, 8)])
def test_delta_rule_by_chunks(ops, chunks, dtype, G, H, d, dv):
    g = torch.Generator().manual_seed(d)
    ins = [delta_inputs(g, n, G, H, d, dv, dtype) for n in LENGTHS]
    a_log, dt_bias = ins[0][2], ins[0][3]
    a_log[0] = 3.0                                          # a head that forgets at once: products of decays that vanish
    state = torch.full((4, H * dv * d + (3 if dv == 36 else 0)), float("nan"), device="cuda")

    def step(o, parts, batch):
        ops.delta_rule(o, rows(parts, [i[0] for i in ins]), rows(parts, [i[1] for i in ins]), dev(a_log), dev(dt_bias), state,
                       batch, G, H, d, dv)

    for got, (qkv, ba, _, _) in zip(walk(step, H * dv, state, LENGTHS, CUTS), ins):
        torch.testing.assert_close(got.to(F64), plain_delta(qkv, ba, a_log, dt_bias, G, H, d, dv), **TOL)


@pytest.mark.parametrize("H,P,N,G", [(8, 64, 128, 1), (4, 20, 64, 2), (3, 36, 100, 3), (10, 8, 16, 1)])
def test_ssd_scan_by_chunks(ops, chunks, H, P, N, G):
    g = torch.Generator().manual_seed(N)
    dt_bias, a_log = torch.randn(H, generator=g) * 0.5, torch.rand(H, generator=g) * 1.5 - 1.0
    a_log[0] = 3.0
    skip = 1 + torch.randn(H, generator=g) * 0.2
    xs = [torch.randn(n, H * P + 2 * G * N, generator=g) for n in LENGTHS]
    dts = [torch.randn(n, H, generator=g) for n in LENGTHS]
    state = torch.full((4, H * P * N), float("nan"), device="cuda")

    def step(o, parts, batch):
        ops.ssd_scan(o, rows(parts, xs), rows(parts, dts), dev(dt_bias), dev(a_log), dev(skip), state, batch, H, P, N, G)

    for got, x, dt in zip(walk(step, H * P, state, LENGTHS, CUTS), xs, dts):
        want = plain_ssd(x, dt, dt_bias, a_log, skip, H, P, N, G)
        # sums over state rows of unit products: relative to the largest of them
        torch.testing.assert_close(got.to(F64), want, rtol=5e-5, atol=1e-5 * want.abs().max().item())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,d,dv,spread", [(2, 128, 256, 4.0), (3, 64, 20, 8.0), (1, 100, 36, 1.0), (2, 8, 16, 3.0)])
def test_mlstm_by_chunks(ops, chunks, dtype, H, d, dv, spread):
    check_mlstm(ops, dtype, H, d, dv, spread, LENGTHS, CUTS)


def scans(ops, kind, H, d, dv, T, g, slower=0.0):
    """One request of T tokens through one of the three scans: (its inputs, a function of them and of whether the sums are to
    be in a fixed order, the plain recurrence in 64 bits, the places of q, k and v in a row of the first input)."""
    if kind == "delta":
        qkv, ba, a_log, dt_bias = delta_inputs(g, T, H, H, d, dv, torch.float32)
        a_log -= slower

        def run(ins, fixed):
            o, state = torch.empty(T, H * dv, device="cuda"), torch.zeros(1, H * d * dv, device="cuda")
            ops.delta_rule(o, dev(ins[0]), dev(ins[1]), dev(a_log), dev(dt_bias), state, step_batch([T], [0], [0]), H, H, d, dv,
                           fixed_order=fixed)
            return o.cpu()
        return (qkv, ba), run, lambda ins: plain_delta(*ins, a_log, dt_bias, H, H, d, dv), (0, H * d, 2 * H * d)
    if kind == "ssd":
        dt_bias, a_log, skip = torch.randn(H, generator=g) * 0.5, torch.rand(H, generator=g) * 1.5 - 1.0 - slower, torch.ones(H)
        xbc, dt = torch.randn(T, H * dv + 2 * d, generator=g), torch.randn(T, H, generator=g)

        def run(ins, fixed):
            y, state = torch.empty(T, H * dv, device="cuda"), torch.zeros(1, H * d * dv, device="cuda")
            ops.ssd_scan(y, dev(ins[0]), dev(ins[1]), dev(dt_bias), dev(a_log), dev(skip), state, step_batch([T], [0], [0]),
                         H, dv, d, 1, fixed_order=fixed)
            return y.cpu()
        return (xbc, dt), run, lambda ins: plain_ssd(*ins, dt_bias, a_log, skip, H, dv, d, 1), (H * dv + d, H * dv, 0)
    proj, gates = mlstm_inputs(g, T, H, d, dv, torch.float32, 4.0)
    proj = proj[:, :-3].contiguous()
    bias = torch.cat((torch.randn(H, generator=g), 2 + torch.randn(H, generator=g)))

    def run(ins, fixed):
        o, state = torch.empty(T, H * dv, device="cuda"), torch.zeros(1, ops.mlstm_state_floats(H, d, dv), device="cuda")
        ops.mlstm_scan(o, dev(ins[0]), dev(ins[1]), dev(bias), 15.0, state, step_batch([T], [0], [0]), H, d, dv, fixed_order=fixed)
        return o.cpu()
    return (proj, gates), run, lambda ins: plain_scan(*ins, bias, 15.0, H, d, dv), (0, H * d, 2 * H * d)


@pytest.mark.parametrize("kind", ["delta", "ssd", "mlstm"])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_a_value_that_is_no_number_stays_with_its_token_and_later_ones(ops, chunks, kind, bad):
    """At every place of a group of four tokens, in q, k, v and the gates: what comes before keeps its bits, and a bad value
    of v keeps to its column."""
    H, d, dv, T = 2, 64, 20, 70
    ins, run, _, (q, k, v) = scans(ops, kind, H, d, dv, T, torch.Generator().manual_seed(3))
    clean = run(ins, False)
    assert torch.isfinite(clean).all()
    for token in (1, 34, 47, 68):
        for which, col in ((0, q), (0, k), (0, v), (1, 0), (1, ins[1].shape[1] - 1)):
            broken = [t.clone() for t in ins]
            broken[which][token, col] = bad
            got = run(broken, False)
            assert torch.equal(got[:token], clean[:token]), (token, which, col)
            if which == 0 and col == v:
                assert not torch.isfinite(got[token, 0]) and torch.equal(got[:, 1:], clean[:, 1:])
            if which == 0 and col == q:
                assert torch.equal(got[token + 1:], clean[token + 1:])


@pytest.mark.parametrize("kind,slower", [("delta", 0.0), ("delta", 4.0), ("ssd", 0.0), ("ssd", 4.0), ("mlstm", 0.0)])
@pytest.mark.parametrize("H,d,dv", [(4, 128, 128), (4, 64, 64), (8, 16, 32)])
def test_error_by_chunks_is_no_larger_than_by_tokens(ops, chunks, kind, slower, H, d, dv):
    """Of 1,024 tokens (``slower``: decays near 1, so that many tokens add up).  The middle one of the tokens' errors: the mLSTM's
    largest come from a few tokens whose normaliser cancels, and differ by chance."""
    ins, run, plain, _ = scans(ops, kind, H, d, dv, 1024, torch.Generator().manual_seed(d), slower)
    want = plain(ins)
    by_chunks, by_tokens = (((run(ins, fixed).to(F64) - want).norm(dim=-1) / want.norm(dim=-1)).median() for fixed in (False, True))
    assert by_chunks <= by_tokens, (by_chunks, by_tokens)
