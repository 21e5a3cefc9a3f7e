"""Vectorised and split kernels at the sizes where they can go wrong: ends of tiles, remainders, the
smallest and largest of their ranges and the forms that fall back to the general kernels.

Each is compared with a 64-bit PyTorch statement of the same operation.  ``BF16`` is the largest
relative error of one rounding to bf16 (half a unit in the last of its 8 bits, 2^-8): a result rounded once
is within it, one that is built from an intermediate rounded once within twice that.
"""
import ctypes
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

BF16 = 2.0 ** -8


def _rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-30)).item()


def _bf16(*shape, seed=0, scale=1.0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, generator=gen, device="cuda") * scale).bfloat16()


# ------------------------------------------------------------------------------ attention backward: 64-row blocks in pairs
@pytest.mark.parametrize("d,hq,hkv", [(128, 4, 1), (64, 3, 1), (128, 2, 2)])
@pytest.mark.parametrize("lengths", [[128], [64, 64], [192, 64, 128], [320, 64], [32, 416, 64, 256]])
def test_attention_gradients_with_odd_numbers_of_blocks(cuda_lib, d, hq, hkv, lengths):
    """Runs whose key tiles see an odd number of 64-query blocks: the last half tile repeats a block, masked, and
    with several heads a tile holds blocks of two heads."""
    from causal_trainer_dev_b200.ops import attention as A

    s = sum(lengths)
    seg = torch.cat([torch.full((n,), i + 1) for i, n in enumerate(lengths)]).int().cuda()[None]
    q, k, v, do = (_bf16(1, s, h, d, seed=i) for i, h in enumerate((hq, hkv, hkv, hq)))
    meta = A.build_attention_meta(seg)
    o, lse = A.flash_attention_forward(q, k, v, meta)
    dq, dk, dv = A.flash_attention_backward(q, k, v, o, do, lse, meta)
    qd, kd, vd = (t.double().requires_grad_() for t in (q, k, v))
    group = hq // hkv
    score = torch.einsum("bqhd,bkhd->bhqk", qd, kd.repeat_interleave(group, 2)) / math.sqrt(d)
    score = score.masked_fill(~A.visibility_mask(seg)[:, None], -math.inf)
    ref = torch.einsum("bhqk,bkhd->bqhd", score.softmax(-1), vd.repeat_interleave(group, 2))
    ref.backward(do.double())
    # P and dS are rounded to bf16 before the products and the results once more
    for got, want in ((o, ref), (dq, qd.grad), (dk, kd.grad), (dv, vd.grad)):
        assert _rel(got, want) < 3 * BF16
    assert _rel(lse, score.logsumexp(-1)) < 1e-6
    assert cuda_lib.device_status() == (0, 0, 0, 0)


def test_attention_keeps_nan_and_stays_finite_elsewhere(cuda_lib):
    """A NaN query makes its own output row NaN and no other."""
    from causal_trainer_dev_b200.ops import attention as A

    q, k, v = (_bf16(1, 512, h, 128, seed=i) for i, h in enumerate((2, 1, 1)))
    q[0, 300, 1] = math.nan
    o, lse = A.flash_attention_forward(q, k, v, A.build_attention_meta(torch.ones(1, 512, dtype=torch.int32, device="cuda")))
    bad = torch.isnan(o).any(-1)
    assert bad[0, 300, 1] and int(bad.sum()) == 1
    assert bool(torch.isnan(o[0, 300, 1]).all())


@pytest.mark.parametrize("d", [128, 64])
@pytest.mark.parametrize("key", [6, 7, 14, 79, 126, 127, 5, 128 + 54])
def test_a_nan_key_reaches_every_query_that_sees_it(cuda_lib, d, key):
    """The scores of one key are NaN, the maxima of the rows stay finite, so query tiles that see the key's whole tile
    take the path whose exponentials of columns 6 and 7 of every 8 run on the FMA pipe (both halves of a pair are
    here, and columns of the ex2 unit): NaN passes through either, and only to queries at or behind the key."""
    from causal_trainer_dev_b200.ops import attention as A

    s = 640
    q, k, v = (_bf16(1, s, h, d, seed=i) for i, h in enumerate((2, 1, 1)))
    k[0, key, 0, 3] = math.nan
    o, _ = A.flash_attention_forward(q, k, v, A.build_attention_meta(torch.ones(1, s, dtype=torch.int32, device="cuda")))
    sees = (torch.arange(s, device="cuda") >= key)[None, :, None]
    assert torch.equal(torch.isnan(o).any(-1), sees.expand(1, s, 2)) and torch.equal(torch.isnan(o).all(-1), sees.expand(1, s, 2))


@pytest.mark.parametrize("d", [128, 64, 96])
@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 33, 3), (1, 128, 28), (2, 6149, 1), (3, 4099, 3), (1, 945, 26), (1, 3001, 9),
                                   (1, 2051, 12), (3, 2049, 4), (1, 945, 28), (1, 1027, 31), (1, 427, 12)])
def test_attention_backward_statistics(cuda_lib, d, shape):
    """A warp per row below 192 d rows (and for other head sizes), above it blocks of 32 tokens and 4 heads, cut off."""
    from causal_trainer_dev_b200.ops import elementwise as E

    b, s, h = shape
    o, do = _bf16(b, s, h, d, seed=1), _bf16(b, s, h, d, seed=2)
    lse = torch.randn(b, h, s, device="cuda")
    neg_lse2, neg_delta = E.attention_backward_stats(o, do, lse)
    assert torch.allclose(neg_lse2, -lse * math.log2(math.e), rtol=1e-6)
    want = -(o.double() * do.double()).sum(-1).permute(0, 2, 1)
    assert (neg_delta.double() - want).abs().max() < 1e-5 * math.sqrt(d)      # fp32 sums of d products of size 1


# ------------------------------------------------------------------------------ memory-bound kernels
@pytest.mark.parametrize("style", ["gpt-neox", "gpt-j"])
@pytest.mark.parametrize("d,rot", [(128, 128), (64, 64), (128, 32), (128, 48), (80, 40), (128, 8), (128, 4)])
@pytest.mark.parametrize("t,heads", [(37, 5), (2051, 5), (601, 29), (16500, 1)])
def test_rope_of_whole_and_partial_vectors(cuda_lib, style, d, rot, t, heads):
    """A thread per pair for few vectors, lanes that walk the heads of a token for many, and warps that share a token's
    heads where there are few tokens."""
    from causal_trainer_dev_b200.ops import elementwise as E

    x = _bf16(t, (heads + 1) * d, seed=3)
    pos = torch.randint(0, 5000, (t,), device="cuda")
    cos, sin = E.rope_table(pos, E.inverse_frequencies(rot, 1e4, device="cuda"))
    for inverse in (False, True):
        got = x.clone()
        E.rope_inplace(got, cos, sin, heads, d, rot, style, inverse=inverse)
        want = E.rope_reference(x[:, :heads * d].reshape(t, heads, d).double().float(), cos, sin, rot, style, inverse)
        assert _rel(got[:, :heads * d].reshape(t, heads, d), want) < BF16
        assert torch.equal(got[:, heads * d:], x[:, heads * d:])              # the columns behind are not touched
        assert torch.equal(got.view(t, heads + 1, d)[:, :heads, rot:], x.view(t, heads + 1, d)[:, :heads, rot:])


@pytest.mark.parametrize("rows", [1, 3, 700])
@pytest.mark.parametrize("d", [8, 2048, 2056, 4096, 4104, 8200, 16384])
def test_rmsnorm_backward_widths(cuda_lib, rows, d):
    from causal_trainer_dev_b200.ops import elementwise as E

    x, dy, res, w = _bf16(rows, d, seed=1), _bf16(rows, d, seed=2), _bf16(rows, d, seed=3), _bf16(d, seed=4)
    _, rstd, _ = E.rmsnorm_forward(x, w, 1e-6)
    xd, wd = x.double().requires_grad_(), w.double().requires_grad_()
    (xd * torch.rsqrt(xd.square().mean(1, keepdim=True) + 1e-6) * wd).backward(dy.double())
    for with_res in (True, False):
        dx, dw = E.rmsnorm_backward(dy, x, w, rstd, dres=res if with_res else None)
        assert _rel(dx, xd.grad + (res.double() if with_res else 0)) < BF16
        assert _rel(dw, wd.grad) < 1e-5                                       # fp32 sums over the rows


@pytest.mark.parametrize("rows,f", [(1, 8), (2, 2048), (7, 2056), (1301, 688), (40003, 24), (4099, 6008)])
def test_swiglu_ragged(cuda_lib, rows, f):
    from causal_trainer_dev_b200.ops import elementwise as E

    gu, dh = _bf16(rows, 2 * f, seed=1, scale=4.0), _bf16(rows, f, seed=2)
    gu[0, :4] = torch.tensor([90.0, -90.0, 0.0, -1e30]).bfloat16().cuda()     # ends of the sigmoid
    gd = gu.double().requires_grad_()
    want = torch.nn.functional.silu(gd[:, :f]) * gd[:, f:]
    want.backward(dh.double())
    assert _rel(E.swiglu_forward(gu), want) < 2 * BF16                        # silu is rounded before the product
    assert _rel(E.swiglu_backward(gu, dh), gd.grad) < BF16


def test_swiglu_of_large_negative_gates(cuda_lib):
    """Every bf16 gate from -88.5 to -64 has a result that bf16 can hold, also where 1 + exp(-gate) is above
    2^126.  (Below -88.7 exp(-gate) is infinite in fp32 and the result zero.)"""
    from causal_trainer_dev_b200.ops import elementwise as E

    gate = -torch.arange(64, 89, 0.5).bfloat16()
    gate = torch.cat([gate, gate.new_zeros(-gate.numel() % 8)]).cuda()
    up, dh = torch.full_like(gate, 3.0), torch.full_like(gate, 0.5)
    gd, ud = gate.double().requires_grad_(), up.double().requires_grad_()
    want = torch.nn.functional.silu(gd) * ud
    want.backward(dh.double())
    gu = torch.cat([gate, up])[None]
    # element by element; __expf is off by up to 2 + 1.2 |x| units in the last place of fp32: 1.3e-5 at 88
    near = lambda got, ref, roundings: bool(((got.double() - ref).abs() <= (roundings * BF16 + 2e-5) * ref.abs()).all())  # noqa: E731
    assert near(E.swiglu_forward(gu)[0], want.detach(), 2)                    # silu is rounded before the product
    dgate, dup = E.swiglu_backward(gu, dh[None])[0].chunk(2)
    assert near(dgate, gd.grad, 1) and near(dup, ud.grad, 1)


def test_swiglu_quotient_of_every_gate(cuda_lib):
    """All 65536 gates of bf16, among themselves (vectors of gates below 87 take the corrected quotient) and each in a vector with a
    gate of 88 (which divides): the same bits, with several factors forward and backward."""
    from causal_trainer_dev_b200.ops import elementwise as E

    gates = torch.arange(-2 ** 15, 2 ** 15, device="cuda").to(torch.int16).view(torch.bfloat16)
    small = gates[gates.abs() < 87]
    large = gates[~(gates.abs() < 87)]                         # infinities and what is not a number among them
    assert small.numel() > 34000 and small.numel() % 4 == large.numel() % 4 == 0
    gen = torch.Generator(device="cuda").manual_seed(9)
    for turn in range(24):
        up, dh = (torch.randn(gates.numel(), generator=gen, device="cuda").bfloat16() for _ in range(2))
        if turn == 0:
            up, dh = torch.ones_like(up), torch.ones_like(dh)

        def run(g, u, d):                                      # rows of 512 gates and their factors
            rows = -(-g.numel() // 512)
            def block(x, fill):
                out = torch.full((rows * 512,), fill, dtype=torch.bfloat16, device="cuda")
                out[:x.numel()] = x
                return out.view(rows, 512)
            gu = torch.cat([block(g, 0.5), block(u, 1.0)], dim=1)
            h, dgu = E.swiglu_forward(gu), E.swiglu_backward(gu, block(d, 1.0))
            return [x.reshape(-1)[:g.numel()] for x in (h, dgu[:, :512], dgu[:, 512:])]

        n = small.numel()
        short = run(small, up[:n], dh[:n])
        wide = lambda x, fill: torch.cat([x.view(-1, 4), torch.full_like(x.view(-1, 4), fill)], 1).reshape(-1)  # noqa: E731
        long = [x.view(-1, 8)[:, :4].reshape(-1) for x in run(wide(small, 88.0), wide(up[:n], 1.0), wide(dh[:n], 1.0))]
        for a, b in zip(short, long):
            assert torch.equal(a.view(torch.int16), b.view(torch.int16)) and not bool(a.isnan().any())
        # a large gate leaves the others of its vector alone, and is itself what it is alone
        m = large.numel()
        mixed = torch.stack([large.view(-1, 4), small[-m:].view(-1, 4)], 2).reshape(-1)
        factor = lambda x: torch.stack([x[:m].view(-1, 4), x[n - m:n].view(-1, 4)], 2).reshape(-1)  # noqa: E731
        got = run(mixed, factor(up), factor(dh))
        alone = run(large, up[:m], dh[:m])
        for a, b, c in zip(got, alone, short):
            a = a.view(-1, 4, 2)
            assert torch.equal(a[:, :, 1].reshape(-1), c[n - m:]) and torch.equal(a[:, :, 0].reshape(-1).nan_to_num(7.0), b.nan_to_num(7.0))


@pytest.mark.parametrize("t", [1497, 1499, 2496, 2497, 4099])      # 128 MiB of traffic: backward above 1497 rows, forward above 2496
def test_swiglu_grids_beyond_l2(cuda_lib, t):
    """Calls on both sides of the sizes where the grids change; vectors with gates whose exponential leaves the range of the short
    division beside others (below -88.7 it is infinite in fp32 and the result zero, as in the long one)."""
    from causal_trainer_dev_b200.ops import elementwise as E

    f = 8960
    gu, dh = _bf16(t, 2 * f, seed=t, scale=4.0), _bf16(t, f, seed=2)
    gu[-1, :40:2] = -torch.arange(70, 90).bfloat16()
    gu[-1, f:f + 40] = 3.0                                   # (products that bf16 holds to its full precision)
    gd = gu.double().requires_grad_()
    want = torch.nn.functional.silu(gd[:, :f]) * gd[:, f:]
    want.backward(dh.double())
    got, dgu = E.swiglu_forward(gu), E.swiglu_backward(gu, dh)
    assert _rel(got, want) < 2 * BF16 and _rel(dgu, gd.grad) < BF16
    # element by element, where the gate is above -88.7: silu is rounded before the product, __expf is off by 1.3e-5 at 88
    near = (got[-1, :40].double() - want[-1, :40]).abs() <= (2 * BF16 + 2e-5) * want[-1, :40].abs()
    assert bool((near | (gu[-1, :40] < -88.6)).all()) and not bool(got.isnan().any()) and not bool(dgu.isnan().any())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n,offset", [(1, 0), (7, 0), (4099, 0), (4099, 1), (1 << 20, 0), ((1 << 20) + 5, 3)])
def test_sum_of_squares_tails_and_alignment(cuda_lib, dtype, n, offset):
    from causal_trainer_dev_b200.ops import elementwise as E

    x = _bf16(n + offset, seed=5).to(dtype)
    x = (x if dtype == torch.bfloat16 else x * 1.001)[offset:]
    assert abs(float(E.sum_of_squares(x)) / float(x.double().square().sum()) - 1) < 1e-5
    if dtype == torch.float32:
        rounded = x.bfloat16().double().square().sum()
        assert abs(float(E.sum_of_squares(x, round_bf16=True)) / float(rounded) - 1) < 1e-5


@pytest.mark.parametrize("rows,n", [(1, 8), (7, 264), (1000, 2048), (5000, 72)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_column_sums(cuda_lib, rows, n, dtype):
    from causal_trainer_dev_b200.ops import elementwise as E

    x = _bf16(rows, n + 8, seed=1)[:, :n]
    first = _bf16(n, seed=2).to(dtype)
    for accumulate in (False, True):
        out = first.clone()
        E.column_sum(x, out, accumulate)
        want = x.double().sum(0) + (first.double() if accumulate else 0)
        assert _rel(out, want) < (BF16 if dtype == torch.bfloat16 else 1e-5)


@pytest.mark.parametrize("rows", [1, 31, 33, 300])
@pytest.mark.parametrize("vocab", [128, 2056, 16400])
def test_cross_entropy_statistics_over_slabs(cuda_lib, rows, vocab):
    from causal_trainer_dev_b200.ops import cross_entropy as CE

    h, w = _bf16(rows, 64, seed=1), _bf16(vocab, 64, seed=2)
    tgt = torch.randint(0, vocab, (rows,), device="cuda")
    wt = torch.rand(rows, device="cuda")
    wt[0] = 0
    nll, total, lse, coef = CE.cut_ce_forward(h, w, tgt, wt, 0.5)
    logits = h.double() @ w.double().t()
    want = logits.logsumexp(1)
    assert (lse.double() - want).abs().max() < 2e-5
    assert torch.allclose(coef, wt * 0.5)
    each = (want - logits.gather(1, tgt[:, None])[:, 0]) * wt.double()
    assert abs(float(nll) - float(each.sum())) < 1e-5 * max(1.0, float(each.abs().sum()))
    assert abs(float(total) - float(wt.double().sum())) < 1e-5 * rows


@pytest.mark.parametrize("d", [8, 6, 264, 1536])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_embedding_gradient_of_long_and_short_runs(cuda_lib, d, dtype):
    """Ids that occur once, up to the length that one warp takes (16), just above it and thousands of times."""
    from causal_trainer_dev_b200.ops import elementwise as E

    counts = {3: 1, 5: 2, 6: 16, 7: 17, 9: 64, 11: 2500, 1: 40, 120: 9, 126: 300}
    ids = torch.cat([torch.full((n,), i) for i, n in counts.items()])
    ids = ids[torch.randperm(ids.numel(), generator=torch.Generator().manual_seed(1))].cuda()
    dout = _bf16(ids.numel(), d, seed=2)
    lo, rows = 2, 120                                                         # ids 1 and 126 belong to another shard
    grad = _bf16(rows, d, seed=3).to(dtype)
    want = grad.double()
    mine = (ids >= lo) & (ids < lo + rows) & (ids != 9)                       # 9: the padding id
    want.index_add_(0, ids[mine] - lo, dout[mine].double())
    first = grad.clone()
    E.embedding_backward(ids, dout, first, 9, lo)
    assert _rel(first, want) < (BF16 if dtype == torch.bfloat16 else 1e-5)
    untouched = torch.ones(rows, dtype=torch.bool, device="cuda")
    untouched[ids[mine] - lo] = False
    assert torch.equal(first[untouched], grad[untouched])
    again = grad.clone()
    E.embedding_backward(ids, dout, again, 9, lo)
    assert torch.equal(first, again)


@pytest.mark.parametrize("tokens", [1, 7, 8, 9, 16, 17, 18, 24, 25, 33, 100])
@pytest.mark.parametrize("kind", ["one", "distinct", "pairs", "tail"])
def test_embedding_gradient_at_the_ends_of_a_block(cuda_lib, tokens, kind):
    """Runs that end with the tokens, fill a block of 8 positions or cross into the next; and a table whose base is not
    16-byte aligned, which the kernel takes two columns at a time."""
    from causal_trainer_dev_b200.ops import elementwise as E

    at = torch.arange(tokens, device="cuda")
    ids = {"one": at * 0 + 3, "distinct": at, "pairs": at // 2, "tail": (at - (tokens - 17)).clamp(max=0) + 20}[kind]
    ids = ids[torch.randperm(tokens, generator=torch.Generator(device="cuda").manual_seed(2), device="cuda")]
    keep = (ids >= 1) & (ids < 65)
    dout = _bf16(tokens, 40, seed=1)
    for offset in (0, 4):
        flat = _bf16(64 * 40 + offset, seed=2)
        grad = flat[offset:].view(64, 40)
        want = grad.double()
        want.index_add_(0, ids[keep] - 1, dout[keep].double())
        E.embedding_backward(ids, dout, grad, -1, 1)
        assert _rel(grad, want) < BF16
        assert torch.equal(flat[:offset], _bf16(64 * 40 + offset, seed=2)[:offset])


# ------------------------------------------------------------------------------ split-K products
@pytest.mark.parametrize("m,n,k", [(1, 8, 2048), (128, 256, 1024), (129, 264, 4104), (70, 130, 9000), (333, 1536, 8200),
                                   (64, 1000, 640), (500, 96, 5000), (1000, 1536, 3000)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
def test_products_with_few_tiles(cuda_lib, m, n, k, a_mn, b_mn):
    """Against 64 bits and against the persistent kernel (which a call that limits its CTAs always gets).  Two of
    the shapes are just too short for the cluster kernel."""
    from causal_trainer_dev_b200.ops.gemm import gemm

    form = ctypes.c_int(), ctypes.c_int()
    planned = cuda_lib.lib().ctb_gemm_split_choice(m, n, k, ctypes.byref(form[0]), ctypes.byref(form[1]))
    assert planned == int((m, n, k) not in [(128, 256, 1024), (64, 1000, 640)])
    pad = lambda x: -(-x // 8) * 8  # noqa: E731
    a = _bf16(k, pad(m), seed=1)[:, :m] if a_mn else _bf16(m, pad(k), seed=1)[:, :k]
    b = _bf16(k, pad(n), seed=2)[:, :n] if b_mn else _bf16(n, pad(k), seed=2)[:, :k]
    want = (a.double().t() if a_mn else a.double()) @ (b.double() if b_mn else b.double().t())
    bias = _bf16(n, seed=3)
    wide = torch.full((m, pad(n) + 8), 7.0, dtype=torch.bfloat16, device="cuda")
    out = gemm(a, b, a_mn=a_mn, b_mn=b_mn, out=wide[:, :n])
    assert _rel(out, want) < BF16
    assert torch.all(wide[:, n:] == 7.0)                                      # nothing beyond column n
    assert _rel(out, gemm(a, b, a_mn=a_mn, b_mn=b_mn, out=torch.empty_like(wide)[:, :n], max_ctas=148)) < 2 * BF16
    assert torch.equal(out, gemm(a, b, a_mn=a_mn, b_mn=b_mn, out=torch.empty_like(wide)[:, :n]))
    biased = gemm(a, b, a_mn=a_mn, b_mn=b_mn, out=torch.empty_like(wide)[:, :n], bias=bias, alpha=0.5)
    assert _rel(biased, (want + bias.double()) * 0.5) < BF16
    full = torch.empty(m, pad(n), dtype=torch.float32, device="cuda")[:, :n]
    assert _rel(gemm(a, b, a_mn=a_mn, b_mn=b_mn, out=full, alpha=0.5), want * 0.5) < 1e-5     # fp32 sums of 9000 products
    assert cuda_lib.device_status() == (0, 0, 0, 0)


@pytest.mark.parametrize("width,slices", [(w, s) for w in (128, 256) for s in (2, 4, 8)])
@pytest.mark.parametrize("m,n,k", [(1, 8, 512), (130, 270, 1000), (257, 512, 520), (300, 131, 4104)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
def test_every_form_of_the_cluster_kernel(cuda_lib, width, slices, m, n, k, a_mn, b_mn):
    """Slices of unequal length, the last k-block, rows and columns cut off, and slices of a single k-block."""
    pad = lambda x: -(-x // 8) * 8  # noqa: E731
    a = _bf16(k, pad(m), seed=1)[:, :m] if a_mn else _bf16(m, pad(k), seed=1)[:, :k]
    b = _bf16(k, pad(n), seed=2)[:, :n] if b_mn else _bf16(n, pad(k), seed=2)[:, :k]
    want = (a.double().t() if a_mn else a.double()) @ (b.double() if b_mn else b.double().t())
    bias, p, ln = _bf16(n, seed=3), cuda_lib.ptr, ctypes.c_long

    def run(dtype, alpha, bias):
        out = torch.full((m, pad(n) + 8), 7.0, dtype=dtype, device="cuda")
        cuda_lib.check(cuda_lib.lib().ctb_gemm_split(
            p(a), p(b), p(out), m, n, k, ln(a.stride(0)), ln(b.stride(0)), ln(out.stride(0)), int(a_mn), int(b_mn),
            int(dtype == torch.float32), ctypes.c_float(alpha), p(bias), width, slices, cuda_lib.stream_ptr()), "ctb_gemm_split")
        assert torch.all(out[:, n:] == 7.0)                                   # nothing beyond column n
        return out[:, :n]

    assert _rel(run(torch.bfloat16, 1.0, None), want) < BF16
    assert _rel(run(torch.bfloat16, 0.5, bias), (want + bias.double()) * 0.5) < BF16
    assert _rel(run(torch.float32, 0.5, None), want * 0.5) < 1e-5             # fp32 sums of 4104 products
    assert cuda_lib.device_status() == (0, 0, 0, 0)


@pytest.mark.parametrize("side", ["weight", "activation"])
@pytest.mark.parametrize("m,n,k", [(64, 1536, 8960), (512, 512, 8192)])
def test_a_product_of_a_gathered_operand_does_not_depend_on_how_far_its_gather_has_come(cuda_lib, side, m, n, k):
    """With chunk flags (the gather may still run) and without (it was seen to be done) the bits are the same."""
    from causal_trainer_dev_b200.ops import gemm as G

    a, b = _bf16(m, k, seed=1), _bf16(n, k, seed=2)
    buffer = b if side == "weight" else a
    src = G.FlagSource(buffer, torch.ones(buffer.numel() // 65536 + 1, dtype=torch.int32, device="cuda"), 65536)
    src.epoch = 1
    G.register_flag_source(src)
    try:
        running = G.gemm(a, b)
        src.complete = torch.cuda.Event()
        src.complete.record()
        src.complete.synchronize()
        done = G.gemm(a, b)
    finally:
        G.unregister_flag_source(src)
    assert torch.equal(running, done)
    assert _rel(done, a.double() @ b.double().t()) < BF16
    assert cuda_lib.device_status() == (0, 0, 0, 0)


# ------------------------------------------------------------------------------ MoBA router
@pytest.mark.parametrize("d,hq,hkv", [(128, 4, 2), (64, 3, 1)])
@pytest.mark.parametrize("top_k", [1, 2, 9, 10])
def test_router_picks_the_best_blocks(cuda_lib, d, hq, hkv, top_k):
    """Up to nine blocks are ranked by eight lanes per token, more by a warp; documents begin anywhere, so the four
    tokens of a warp may differ in their block or document, or be padding."""
    from causal_trainer_dev_b200.ops import moba as M

    block, lengths = 128, [130, 1301, 37, 2500]
    s = 4096
    seg = torch.zeros(1, s, dtype=torch.int32, device="cuda")
    starts = torch.zeros(1, s, dtype=torch.int32, device="cuda")
    at = 0
    for i, n in enumerate(lengths):
        seg[0, at:at + n], starts[0, at:at + n] = i + 1, at
        at += n
    q, k = _bf16(1, s, hq, d, seed=1), _bf16(1, s, hkv, d, seed=2)
    sel = M.route(q, k, seg, starts, block, top_k)
    bits = torch.stack([(sel[0, :, :, c >> 5] >> (c & 31)) & 1 for c in range(32 * sel.shape[-1])], -1).bool()   # [Hq,S,blocks]
    at = 0
    for n in lengths:
        nb = -(-n // block)
        means = torch.stack([k[0, at + c * block:at + (c + 1) * block].double().mean(0) for c in range(nb)])       # [nb,Hkv,D]
        own = torch.arange(n, device="cuda") // block
        gate = torch.einsum("shd,chd->hsc", q[0, at:at + n].double(), means.repeat_interleave(hq // hkv, 1))
        gate = gate.masked_fill(torch.arange(nb, device="cuda")[None, None] >= own[None, :, None], -math.inf)
        chosen = bits[:, at:at + n, :nb]
        assert not bits[:, at:at + n, nb:].any()
        assert bool(chosen.gather(2, own[None, :, None].expand(hq, n, 1)).all())
        picks = chosen & ~torch.isinf(gate)
        assert torch.equal(picks.sum(-1), own.clamp(max=top_k - 1)[None].expand(hq, n))
        # no block that was left out scores higher than one that was picked (beyond fp32 sums of d products)
        worst = gate.masked_fill(~picks, math.inf).amin(-1)
        left = gate.masked_fill(picks, -math.inf).amax(-1)
        assert bool((left <= worst + 1e-5).all())
        at += n
    assert not bits[:, at:].any()


@pytest.mark.parametrize("s,block,top_k,kinds", [(4096, 128, 3, "bits scan walk"), (1024, 256, 2, "bits scan walk"),
                                                 (192512, 4096, 4, "bits scan"), (192640, 4096, 4, "bits scan walk")])
def test_rank_kernels_group_alike(cuda_lib, monkeypatch, s, block, top_k, kinds):
    """Ranks from a bit per token (rows of up to 192512 tokens), by the scan (longer rows) and by the walk give the same
    grouping bit for bit: documents that begin anywhere, padding between and behind them."""
    from causal_trainer_dev_b200.ops import attention as A
    from causal_trainer_dev_b200.ops import moba as M

    seg = torch.zeros(2, s, dtype=torch.int32, device="cuda")
    for row, cuts in enumerate(([0, s // 37, s // 3 + 5, s - 77], [13, s // 2 + 1, s])):
        for i, (lo, hi) in enumerate(zip(cuts[:-1], cuts[1:])):
            seg[row, lo:hi] = i + 1
    seg[0, s // 3 - 40:s // 3 + 5] = 0                                        # padding between two documents
    q, k = _bf16(2, s, 2, 64, seed=1), _bf16(2, s, 1, 64, seed=2)
    meta = A.build_attention_meta(seg)
    seen = []
    for kind in kinds.split():
        monkeypatch.setenv("CTB_MOBA_RANK", kind)
        g = M.build_groups(q, k, meta, block, top_k)
        seen.append((g.totals, g.row_of, g.pos_of, g.fwd_desc, g.dq_desc, g.dkv_desc))
    assert int(seen[0][0][0]) > 0
    for other in seen[1:]:
        assert all(torch.equal(a, b) for a, b in zip(seen[0], other))
    # ranks: the rows of a (document, head, block) in the order of their tokens
    rows = int(seen[0][0][0])
    token = (seen[0][1][:rows] // 2).long()
    pos = seen[0][2]
    for h in range(2):
        for j in range(top_k - 1):
            mine = pos[0, h, :, j]
            assert torch.equal(token[mine[mine >= 0].long()], torch.nonzero(mine >= 0)[:, 0])
