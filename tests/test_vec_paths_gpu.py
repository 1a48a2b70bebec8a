"""Kernels that take several elements a thread where sizes and addresses allow it, against 64-bit references and against the
same kernels' general form (reached by rows an odd number of elements apart)."""
import pytest
import torch

import plain_muvonex as pm
from test_muvonex_ops_gpu import F64, dev, portions_of, rotary_table, step_batch, tol

pytestmark = pytest.mark.gpu

DTYPES = [torch.float32, torch.bfloat16]


@pytest.fixture(scope="module")
def ops():
    from nanohybrid_vlm_b200.kernels import ops
    return ops


def odd_rows(t):
    """The same values in rows one element further apart."""
    wide = torch.zeros(t.shape[0], t.shape[1] + 1, dtype=t.dtype, device=t.device)
    wide[:, :-1] = t
    return wide[:, :-1]


# groups of 8, 16, 32 and 256 threads, one piece and four; a weight per group, per row, and one that ends inside a group
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("groups,size,period,gate_first", [(5, 64, 64, False), (3, 72, 216, True), (16, 128, 128, False),
                                                           (2, 256, 512, True), (3, 96, 16, True), (1, 264, 264, True),
                                                           (1, 2048, 2048, True), (2, 2056, 4112, False), (1, 8192, 8192, True),
                                                           (1, 8200, 8200, True), (3, 128, 192, False)])
def test_gated_rmsnorm(ops, dtype, groups, size, period, gate_first):
    g = torch.Generator().manual_seed(size)
    T, n = 9, groups * size
    y = torch.randn(T, n, generator=g) * 3
    z = torch.randn(T, n, generator=g).to(dtype)
    w = (1 + 0.2 * torch.randn(period, generator=g)).to(dtype)
    full = w.repeat(n // period) if n % period == 0 else None
    for gate in ("silu", "sigmoid"):
        outs = []
        for zz in (dev(z), odd_rows(dev(z))):
            out = torch.full((T, n), float("nan"), dtype=dtype, device="cuda")
            ops.gated_rmsnorm(out, dev(y), zz, dev(w), groups, 1e-5, gate_first, gate)
            outs.append(out)
        torch.testing.assert_close(outs[0].float(), outs[1].float(), **tol(dtype, bf16=2 ** -7))
    if full is not None:
        ops.gated_rmsnorm(out, dev(y), dev(z), dev(w), groups, 1e-5, gate_first)
        want = pm.gated_norm(y.to(F64), z.to(F64), full.to(F64), groups, 1e-5, gate_first)
        torch.testing.assert_close(out.cpu().to(F64), want, **tol(dtype))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("nq,nkv,dk,dv,rot,opts", [
    (3, 1, 128, 128, 128, {}), (4, 2, 64, 32, 32, dict(weights=True)), (2, 2, 256, 128, 64, dict(norm_first=True, weights=True)),
    (5, 1, 72, 40, 48, dict(eps=None)), (2, 1, 128, 128, 0, dict(bias=True, values_from_keys=True)), (3, 3, 8, 8, 0, {}),
    (2, 1, 96, 96, 40, dict(interleaved=True)), (2, 2, 128, 64, 16, dict(norm_first=True)), (1, 1, 264, 8, 16, {})])
def test_rope_norm_store(ops, dtype, nq, nkv, dk, dv, rot, opts):
    g = torch.Generator().manual_seed(dk + nq)
    opts = dict(opts)
    T, page, n_pages, row = 13, 8, 4, -(-max(dk, dv) // 8) * 8 + 8
    vk = opts.get("values_from_keys", False)
    qkv = torch.randn(T, (nq + nkv) * dk + (0 if vk else nkv * dv), generator=g).to(dtype).cuda()
    kw = dict(norm_first=opts.get("norm_first", False), interleaved=opts.get("interleaved", False), values_from_keys=vk)
    if opts.get("weights"):
        kw.update(q_weight=dev(torch.randn(dk, generator=g).to(dtype)), k_weight=dev(torch.randn(dk, generator=g).to(dtype)))
    if opts.get("bias"):
        kw.update(bias=dev(torch.randn((nq + nkv) * dk, generator=g).to(dtype)))
    table = dev(rotary_table(rot, 10000.0, None, 50)) if rot else None
    pos = torch.randint(0, 50, (T,), generator=g, dtype=torch.int32).cuda()
    slots = torch.randperm(n_pages * page, generator=g)[:T].to(torch.int32)
    slots[4] = -1                                              # stored nowhere
    got = []
    for x in (qkv, odd_rows(qkv)):
        q = torch.full((T, nq * dk), float("nan"), dtype=dtype, device="cuda")
        pages = torch.full((n_pages, 2, nkv, page, row), 7.0, dtype=dtype, device="cuda")
        ops.rope_norm_store(x, q, pages, dev(slots), pos, table, rot, nq, nkv, dk, dv, opts.get("eps", 1e-5), **kw)
        only = torch.full((T, nq * dk), float("nan"), dtype=dtype, device="cuda")
        ops.rope_norm_store(x, only, None, None, pos, table, rot, nq, nkv, dk, dv, opts.get("eps", 1e-5), **kw)
        assert torch.equal(only, q)
        got.append((q.float(), pages.float()))
    # the sum of squares in another order: results may round the other way
    for a, b in zip(*got):
        torch.testing.assert_close(a, b, **tol(dtype, f32=1e-6, bf16=2 ** -7))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("C,K", [(68, 4), (132, 3), (516, 2), (64, 1)])
def test_short_filters_of_long_steps(ops, dtype, C, K):
    """Requests that end inside, at and before a tile of 16 tokens and a piece of four, fresh and with a past."""
    g = torch.Generator().manual_seed(C)
    news, starts, slots = [1, 300, 15, 17, 2, 250, 3], [4, 0, 9, 0, 1, 2, 0], [3, 0, 1, 6, 2, -1, 5]
    T = sum(news)
    x = torch.randn(T, C, generator=g).to(dtype).cuda()
    w, w2 = (dev((torch.randn(C, K, generator=g) * 0.5).to(dtype)) for _ in range(2))
    bias = dev((torch.randn(C, generator=g) * 0.3).to(dtype))
    first = torch.randn(7, max(K - 1, 1) * C, generator=g).cuda()
    got, b = [], step_batch(news, starts, slots)
    for xx in (x, odd_rows(x)):
        s1 = first.clone()
        y32, y = torch.empty(T, C, device="cuda"), torch.empty(T, C, dtype=dtype, device="cuda")
        ops.short_conv_silu(y32, xx, w, bias, s1.clone(), b)
        ops.short_conv_silu(y, xx, w, None, s1, b)
        got.append((y32, y, s1))
    f1, f2, f3 = (torch.empty(T, C, dtype=dtype, device="cuda") for _ in range(3))
    ops.causal_filter_add(f1, f2, x, w, w2, first.clone(), b)
    ops.causal_filter_add(f3, None, x, w, None, first.clone(), b)
    for a, b in zip(*got):
        assert torch.equal(a, b)                               # the same operations in the same order
    # filter_add takes whole rows only: against its definition
    past = torch.zeros(T, C, K - 1, dtype=F64, device="cuda")
    at = 0
    for n, start, slot in zip(news, starts, slots):
        old = (first[slot].view(-1, C)[:K - 1].to(F64) if start > 0 and slot >= 0 and K > 1
               else torch.zeros(K - 1, C, dtype=F64, device="cuda"))
        seq = torch.cat([old, x[at:at + n].to(F64)])
        for j in range(K - 1):
            past[at:at + n, :, j] = seq[j:j + n]
        at += n
    for f, ww in ((f1, w), (f2, w2), (f3, w)):
        want = x.to(F64) * (1 + ww[:, -1].to(F64)) + (past * ww[:, :-1].to(F64)).sum(-1)
        torch.testing.assert_close(f.to(F64), want, **tol(dtype, f32=1e-5))
    assert torch.equal(f1, f3)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("C,K,two", [(68, 4, True), (132, 3, False), (516, 2, True), (64, 1, False)])
def test_filter_add_has_the_same_bits_in_long_and_short_steps(ops, dtype, C, K, two):
    """The same requests in one step of more than 512 tokens (four channels a thread) and in portions of fewer."""
    g = torch.Generator().manual_seed(C)
    lengths = [300, 17, 250]
    xs = [torch.randn(n, C, generator=g).to(dtype).cuda() for n in lengths]
    w, w2 = (dev((torch.randn(C, K, generator=g) * 0.5).to(dtype)) for _ in range(2))
    seen = []
    for cuts in ([[], [], []], [[1, 150], [1, 16], [1, 120]]):
        state = torch.full((3, max(K - 1, 1) * C), float("nan"), device="cuda")
        got = [[] for _ in lengths]
        for who, starts, news in portions_of(lengths, cuts):
            x = torch.cat([xs[r][s:s + n] for r, s, n in zip(who, starts, news)])
            f1, f2 = torch.empty_like(x), torch.empty_like(x)
            ops.causal_filter_add(f1, f2 if two else None, x, w, w2 if two else None, state, step_batch(news, starts, who))
            for r, a, b in zip(who, f1.split(news), f2.split(news)):
                got[r].append(torch.cat([a, b], 1) if two else a)
        seen.append([torch.cat(p) for p in got] + ([state] if K > 1 else []))
    for a, b in zip(*seen):
        assert torch.equal(a, b)


def off_by_one(t):
    """The same values, contiguous, one element behind a boundary of 16 bytes."""
    room = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    room[1:] = t.reshape(-1)
    return room[1:].view(t.shape)


# a warp a row; parts of one and of several warps; odd numbers of warps; the widest row of the vector form, and wider
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("width,groups", [(256, 1), (512, 2), (768, 1), (1280, 5), (2048, 1), (2048, 4), (4096, 2), (8192, 1), (8448, 1)])
@pytest.mark.parametrize("n_addends", [0, 1, 2, 3])
def test_norm_over_the_stream(ops, dtype, width, groups, n_addends):
    """Against 64 bits, and the bits of the form that takes a column at a time: a norm's last bit can tip what follows in 16 bits."""
    g = torch.Generator().manual_seed(width + n_addends)
    T, coefs = 5, (0.7, -1.25, 2.0)
    stream = torch.randn(T, width, generator=g) * 3
    stream[:, :width // groups] *= 50                       # one loud part must not quieten the others
    adds = [torch.randn(T, width, generator=g).to(dtype) for _ in range(n_addends)]
    w = (1 + 0.2 * torch.randn(width, generator=g)).to(dtype)
    want_stream = stream.to(F64) + sum(c * a.to(F64) for c, a in zip(coefs, adds))
    parts = want_stream.view(T, groups, -1)
    want = (parts / (parts.square().mean(-1, keepdim=True) + 1e-5).sqrt()).view(T, width) * (w.to(F64) + 0.5)
    for rows in (None, torch.tensor([4, 0, 2], dtype=torch.int32)):
        pick, seen = slice(None) if rows is None else rows.long(), []
        for place in (lambda t: t, off_by_one):
            s, out = place(dev(stream)), place(torch.full((T if rows is None else 3, width), float("nan"), dtype=dtype, device="cuda"))
            ops.rmsnorm_stream(out, s, place(dev(w)), 1e-5, [(place(dev(a)), c) for a, c in zip(adds, coefs)],
                               rows=None if rows is None else dev(rows), weight_offset=0.5, groups=groups)
            torch.testing.assert_close(out.cpu().to(F64), want[pick], **tol(dtype))
            torch.testing.assert_close(s.cpu().to(F64), want_stream if rows is None else stream.to(F64), rtol=1e-6, atol=1e-4)
            seen.append((out.cpu(), s.cpu()))
        assert torch.equal(seen[0][0], seen[1][0]) and torch.equal(seen[0][1], seen[1][1])


# one block across with idle threads, a last block in part, two whole blocks; more rows than blocks down
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("width,T", [(96, 9), (1028, 9), (2048, 3), (512, 1200), (1536, 700)])
def test_dyntanh_over_the_stream(ops, dtype, width, T):
    g = torch.Generator().manual_seed(width)
    pre, post = ([dev(t.to(dtype)) for t in (0.3 + torch.rand(1, generator=g), 1 + 0.3 * torch.randn(width, generator=g),
                                             0.3 * torch.randn(width, generator=g))] for _ in range(2))
    stream, a = torch.randn(T, width, generator=g) * 2, torch.randn(T, width, generator=g).to(dtype)
    rows = torch.randperm(T, generator=g)[:max(1, T - 1)].int()
    f = lambda x, p: torch.tanh(p[0].cpu().to(F64) * x.to(F64)) * p[1].cpu().to(F64) + p[2].cpu().to(F64)     # noqa: E731
    for addend, norm in ((None, None), (a, None), (a, post)):
        for gather in (None, rows):
            pick, seen = slice(None) if gather is None else gather.long(), []
            want_stream = stream.to(F64) + (0 if addend is None else addend.to(F64) if norm is None else f(addend, norm))
            for place in (lambda t: t, off_by_one):
                s, out = place(dev(stream)), place(torch.full((T if gather is None else len(gather), width), float("nan"), dtype=dtype, device="cuda"))
                ops.dyntanh_stream(out, s, tuple(pre), None if addend is None else place(dev(addend)), None if norm is None else tuple(norm),
                                   rows=None if gather is None else dev(gather), write_stream=gather is None)
                torch.testing.assert_close(out.cpu().to(F64), f(want_stream, pre)[pick], **tol(dtype))
                kept = want_stream if gather is None else stream.to(F64)
                torch.testing.assert_close(s.cpu().to(F64), kept, **tol(torch.float32))
                seen.append((out.cpu(), s.cpu()))
            assert torch.equal(seen[0][0], seen[1][0]) and torch.equal(seen[0][1], seen[1][1])


# the three widths of a thread per four columns of each quarter, beside the tests of the other widths above
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("width", [512, 1024, 2048])
@pytest.mark.parametrize("n_addends,gathered", [(0, False), (1, False), (2, True), (3, False)])
def test_norm_over_the_stream_by_quarters_has_the_same_bits(ops, dtype, width, n_addends, gathered):
    g = torch.Generator().manual_seed(width + n_addends)
    T, coefs = 70, (0.7, -1.25, 2.0)
    stream, w = torch.randn(T, width, generator=g) * 3, (1 + 0.2 * torch.randn(width, generator=g)).to(dtype)
    adds = [torch.randn(T, width, generator=g).to(dtype) for _ in range(n_addends)]
    rows, seen = torch.randperm(T, generator=g)[:33].int() if gathered else None, []
    for place in (lambda t: t, off_by_one):
        s, out = place(dev(stream)), place(torch.full((33 if gathered else T, width), float("nan"), dtype=dtype, device="cuda"))
        ops.rmsnorm_stream(out, s, place(dev(w)), 1e-5, [(place(dev(a)), c) for a, c in zip(adds, coefs)],
                           rows=dev(rows) if gathered else None, weight_offset=1.0)
        seen.append((out.cpu(), s.cpu()))
    assert seen[0][0].isfinite().all() and torch.equal(seen[0][0], seen[1][0]) and torch.equal(seen[0][1], seen[1][1])


# pieces of x and w on their way at once: one, two, four and eight, and a second round of each; few and many outputs
@pytest.mark.parametrize("K", [8, 256, 264, 512, 520, 1024, 1032, 2048, 2056, 4104])
@pytest.mark.parametrize("M,N", [(3, 7), (700, 8)])
def test_small_products_with_float32_sums(ops, K, M, N):
    g = torch.Generator().manual_seed(K)
    x, w = torch.randn(M, K, generator=g).bfloat16(), torch.randn(N, K, generator=g).bfloat16()
    out = torch.full((M, N), float("nan"), device="cuda")
    ops.linear_f32(out, dev(x), dev(w))
    want = x.to(F64) @ w.to(F64).T
    size = x.abs().to(F64) @ w.abs().to(F64).T
    # 32-bit sums of exact products: K / 128 of a lane one after the other, then a tree of seven
    assert ((out.cpu().to(F64) - want).abs() <= (K / 128 + 8) * 2 ** -24 * size).all()
