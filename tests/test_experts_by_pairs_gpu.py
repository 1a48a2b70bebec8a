"""The experts' tcgen05 products by pairs of SMs (tiles of 256 rows, 128 in each block) and the ordering by a cluster of
blocks, at the sizes where they can go wrong: runs of rows around a half and a whole tile, output columns around a panel and
around the pieces that a thread writes, inner sizes around a stage."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from nanohybrid_vlm_b200.kernels import ops as module
    return module


# rows of each expert: none, one, around 128 and 256 rows, several tiles with the last one half empty
RUNS = [0, 1, 127, 128, 129, 255, 256, 257, 640, 0]


@pytest.mark.parametrize("gated", [True, False])
@pytest.mark.parametrize("W,ff", [(64, 128), (72, 136), (8, 24), (200, 264), (256, 40), (392, 520)])
def test_products(ops, monkeypatch, gated, W, ff):
    g = torch.Generator().manual_seed(W + ff)
    E, T = len(RUNS), sum(RUNS)
    ids = torch.cat([torch.full((n,), e) for e, n in enumerate(RUNS)])[torch.randperm(T, generator=g)].int()[:, None].cuda()
    x = torch.randn(T, W, generator=g).bfloat16().cuda()
    gate, up = ((torch.randn(E, ff, W, generator=g) / W ** 0.5).bfloat16().cuda() for _ in range(2))
    down = (torch.randn(E, W, ff, generator=g) / ff ** 0.5).bfloat16().cuda()
    scale = (torch.rand(T, 1, generator=g) + 0.5).cuda()
    monkeypatch.setattr(ops, "MOE_TCGEN05", True)
    y, pos = ops.moe_experts(x, gate if gated else None, up, down, ids, 1.5, 1.702, 1.0, scale)
    ops.raise_wait_errors()
    assert sorted(pos.tolist()) == sorted(set(pos.tolist())) and pos.min() >= 0
    got = y[pos.long()].double()
    for e in range(E):
        at = (ids[:, 0] == e).nonzero()[:, 0]
        # the sums are rounded to bfloat16 before the unit and the unit's result before the second product, as in the kernel
        s = scale[at].double()
        u = (s * (x[at].double() @ up[e].double().T)).bfloat16().double()
        if gated:
            v = (s * (x[at].double() @ gate[e].double().T)).bfloat16().double().clamp(max=1.5)
            a = v * torch.sigmoid(1.702 * v) * (u.clamp(-1.5, 1.5) + 1.0)
        else:
            a = torch.relu(u) ** 2
        want = a.bfloat16().double() @ down[e].double().T
        # one result: half a unit of bfloat16 (2^-9) from the last rounding; a 32-bit sum that falls on the other side of a
        # rounding moves one of ff terms by 2^-8 of itself: well under 2^-7 of the largest result
        torch.testing.assert_close(got[at], want, rtol=2 ** -8, atol=2 ** -7 * max(1.0, want.abs().max().item() if len(at) else 0))


def test_padding_rows_that_hold_no_numbers(ops, monkeypatch):
    """The rows of padding are not written by the gather, and whatever they hold stays in their own rows."""
    g = torch.Generator().manual_seed(0)
    x = torch.randn(140, 64, generator=g).bfloat16().cuda()
    up = torch.randn(2, 64, 64, generator=g).bfloat16().cuda()
    ids = (torch.arange(140) >= 130).int()[:, None].cuda()           # 130 rows: two of the upper half; 10 rows: no upper half
    sorted_slots, pos, tile_expert = ops.moe_align(ids, 2, 256)
    assert tile_expert.tolist()[:2] == [0, 1] and set(tile_expert.tolist()[2:]) <= {-1}
    rows = sorted_slots.numel()
    xs, out = (torch.full((rows, 64), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    ops.call("nhv_moe_gather_rows", xs.data_ptr(), x.data_ptr(), sorted_slots.data_ptr(), rows, 1, 64, ops.stream_ptr())
    assert torch.equal(xs[pos.long()], x) and xs.isnan().any(-1).sum() == rows - 140
    ops.call("nhv_moe_gemm_tcgen05", 0, out.data_ptr(), xs.data_ptr(), up.data_ptr(), None, 2, sorted_slots.data_ptr(),
             tile_expert.data_ptr(), rows // 256, 64, 64, 0.0, 0.0, 0.0, None, ops.stream_ptr())
    ops.raise_wait_errors()
    want = torch.einsum("tw,tfw->tf", x.double(), up.double()[ids[:, 0].long()])
    torch.testing.assert_close(out[pos.long()].double(), want, rtol=2 ** -8, atol=2 ** -8 * want.abs().max().item())
    assert out.isnan().any(-1).sum() == rows - 140                   # rows of padding are not written


@pytest.mark.parametrize("n,E,tile", [(2048, 7, 16), (2049, 7, 16), (2049, 2048, 64), (5000, 16, 256), (40001, 3, 128),
                                      (8192, 1, 256), (4097, 300, 16)])
def test_ordering(ops, n, E, tile):
    g = torch.Generator().manual_seed(n)
    ids = torch.randint(0, E + 2, (n, 1), generator=g).int()         # the last two are identity choices
    ids[ids == E // 2] = E                                           # an expert that nobody chooses
    slots, pos, tile_expert = (t.cpu() for t in ops.moe_align(ids.cuda(), E, tile))
    at = 0
    for e in range(E):
        mine = (ids[:, 0] == e).nonzero()[:, 0]
        end = at + -(-len(mine) // tile) * tile
        assert sorted(slots[at:at + len(mine)].tolist()) == mine.tolist()
        assert (slots[at + len(mine):end] == -1).all() and (tile_expert[at // tile:end // tile] == e).all()
        at = end
    assert (slots[at:] == -1).all() and (tile_expert[at // tile:] == -1).all()
    real = ids[:, 0] < E
    assert (pos[~real] == -1).all() and torch.equal(slots[pos[real].long()], real.nonzero()[:, 0].int())
