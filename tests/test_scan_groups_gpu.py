"""Scans by chunks with two groups of 16 columns a block (more groups than SMs): columns that leave the second group empty or in
part, heads of less than a kernel's width, requests that end at, before and behind a chunk, values that are no number."""
import pytest
import torch

from test_muvonex_ops_gpu import F64, delta_inputs, dev, plain_delta, plain_ssd, step_batch
from test_nomudra_ops_gpu import mlstm_inputs, plain_scan
from test_scan_paths_gpu import TOL, cancellation, rows, scans, walk

pytestmark = pytest.mark.gpu
LENGTHS = [70, 33, 64, 41]
CUTS = [[33], [1], [32], []]            # per step: 33, 1, 32, 41 tokens; then 37, 32, 32, -


@pytest.fixture(scope="module")
def ops():
    from nanohybrid_vlm_b200.kernels import ops
    return ops


@pytest.fixture(autouse=True)
def chunks(ops):
    ops.CHUNK_SCAN_TOKENS = 16
    yield
    ops.CHUNK_SCAN_TOKENS = 0


@pytest.mark.parametrize("G,H,d,dv", [(7, 14, 128, 48), (20, 20, 100, 20), (5, 40, 64, 16)])
def test_delta_rule(ops, G, H, d, dv):
    g = torch.Generator().manual_seed(d)
    ins = [delta_inputs(g, n, G, H, d, dv, torch.float32) for n in LENGTHS]
    a_log, dt_bias = ins[0][2], ins[0][3]
    state = torch.full((4, H * dv * d), float("nan"), device="cuda")

    def step(o, parts, batch):
        ops.delta_rule(o, rows(parts, [i[0] for i in ins]), rows(parts, [i[1] for i in ins]), dev(a_log), dev(dt_bias), state,
                       batch, G, H, d, dv)

    for got, (qkv, ba, _, _) in zip(walk(step, H * dv, state, LENGTHS, CUTS), ins):
        torch.testing.assert_close(got.to(F64), plain_delta(qkv, ba, a_log, dt_bias, G, H, d, dv), **TOL)


@pytest.mark.parametrize("H,P,N,G", [(14, 48, 128, 1), (20, 20, 36, 4), (40, 16, 64, 2)])
def test_state_space(ops, H, P, N, G):
    g = torch.Generator().manual_seed(N)
    dt_bias, a_log = torch.randn(H, generator=g) * 0.5, torch.rand(H, generator=g) * 1.5 - 1.0
    skip = 1 + torch.randn(H, generator=g) * 0.2
    xs = [torch.randn(n, H * P + 2 * G * N, generator=g) for n in LENGTHS]
    dts = [torch.randn(n, H, generator=g) for n in LENGTHS]
    state = torch.full((4, H * P * N), float("nan"), device="cuda")

    def step(o, parts, batch):
        ops.ssd_scan(o, rows(parts, xs), rows(parts, dts), dev(dt_bias), dev(a_log), dev(skip), state, batch, H, P, N, G)

    for got, x, dt in zip(walk(step, H * P, state, LENGTHS, CUTS), xs, dts):
        want = plain_ssd(x, dt, dt_bias, a_log, skip, H, P, N, G)
        torch.testing.assert_close(got.to(F64), want, rtol=5e-5, atol=1e-5 * want.abs().max().item())


@pytest.mark.parametrize("H,d,dv,spread", [(14, 128, 48, 4.0), (20, 36, 20, 1.0), (40, 64, 16, 8.0)])
def test_mlstm(ops, H, d, dv, spread):
    g = torch.Generator().manual_seed(d)
    ins = [mlstm_inputs(g, n, H, d, dv, torch.bfloat16, spread) for n in LENGTHS]
    ins = [(p[:, :2 * H * d + H * dv].contiguous(), gt) for p, gt in ins]
    bias = torch.cat((torch.randn(H, generator=g), 2 + torch.randn(H, generator=g)))
    floats = ops.mlstm_state_floats(H, d, dv)
    state = torch.full((4, -(-floats // 4) * 4), float("nan"), device="cuda")

    def step(o, parts, batch):
        ops.mlstm_scan(o, rows(parts, [i[0] for i in ins]), rows(parts, [i[1] for i in ins]), dev(bias), 15.0, state, batch,
                       H, d, dv)

    for got, (proj, gates) in zip(walk(step, H * dv, state, LENGTHS, CUTS), ins):
        want = plain_scan(proj, gates, bias, 15.0, H, d, dv)
        # the bound of the scans' other tests: logarithms of gates known to 4e-6, added up over the tokens, and what cancels
        loss = cancellation(proj, gates, bias, H, d)
        off = (got.to(F64) - want).view(-1, H, dv).norm(dim=-1) / want.view(-1, H, dv).norm(dim=-1)
        assert (off <= 6e-5 * (1 + loss)).all(), (off / (1 + loss)).max()
    assert state[:, :floats].isfinite().all()                     # every copy of the normaliser is written


@pytest.mark.parametrize("kind", ["delta", "ssd", "mlstm"])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_a_value_that_is_no_number(ops, kind, bad):
    H, d, dv, T = 40, 64, 64, 70
    ins, run, _, (q, k, v) = scans(ops, kind, H, d, dv, T, torch.Generator().manual_seed(3))
    clean = run(ins, False)
    for token in (1, 34, 68):
        for col in (v, v + 17, v + 40):
            broken = [ins[0].clone(), ins[1]]
            broken[0][token, col] = bad
            got = run(broken, False)
            rest = [i for i in range(H * dv) if i != col - v]
            assert torch.equal(got[:token], clean[:token]) and torch.equal(got[:, rest], clean[:, rest])
            assert not torch.isfinite(got[token, col - v])


@pytest.mark.parametrize("kind", ["delta", "ssd", "mlstm"])
def test_a_value_above_the_largest_bfloat16(ops, kind):
    """A number that a bfloat16 rounds to an infinity: it moves its column from its token on, and nothing before or beside."""
    H, d, dv, T = 40, 64, 64, 70
    ins, run, plain, (q, k, v) = scans(ops, kind, H, d, dv, T, torch.Generator().manual_seed(5))
    ins[0][:, :v] *= 1e-3 if kind != "ssd" else 1           # (no product beyond the range: the sums are numbers)
    if kind == "ssd":
        ins[0][:, H * dv:] *= 1e-3
    clean = run(ins, False)
    for token in (0, 1, 34, 68):
        for col in (v, v + 17, v + 40):
            big = [ins[0].clone(), ins[1]]
            big[0][token, col] = 3.4e38
            got = run(big, False)
            rest = [i for i in range(H * dv) if i != col - v]
            assert torch.equal(got[:token], clean[:token]) and torch.equal(got[:, rest], clean[:, rest])
            # (delta rule: a head may keep more than half of what it holds, so that sums may leave the range)
            if kind == "ssd":
                want = plain(big)[token:, col - v]
                assert ((got[token:, col - v].to(F64) - want).abs() <= 1e-5 * want.abs().max()).all()


@pytest.mark.parametrize("length", [32, 33, 64, 5])
def test_one_product_enters_the_state_as_it_is(ops, length):
    """The last token alone brings a value, at full weight: the state is key times value, exact in 32 bits.  (What is given back to
    sums that the tensor cores cut off stays below half a unit of the last place, so that exact ones stay.)"""
    H, d, dv = 8, 64, 32
    g = torch.Generator().manual_seed(7)
    proj = torch.randn(length, 2 * H * d + H * dv, generator=g)
    proj[:, H * d:2 * H * d] = 2.0 ** torch.randint(-3, 4, (length, H * d), generator=g)
    proj[:-1, 2 * H * d:] = 0
    gates = torch.zeros(length, 2 * H)
    gates[-1, :H] = 40.0                                    # the largest input gate by far: its weight is exp(0)
    state = torch.zeros(1, ops.mlstm_state_floats(H, d, dv), device="cuda")
    o = torch.empty(length, H * dv, device="cuda")
    ops.CHUNK_SCAN_TOKENS = 4
    ops.mlstm_scan(o, dev(proj), dev(gates), dev(torch.zeros(2 * H)), 15.0, state, step_batch([length], [0], [0]), H, d, dv)
    k, v = proj[-1, H * d:2 * H * d].view(H, 1, d), proj[-1, 2 * H * d:].view(H, dv, 1)
    assert torch.equal(state[0, :H * dv * d].view(H, dv, d).cpu(), k * v)
