"""dK / dV of few key tiles: a tile's queries cut over several work items, whose fp32 sums are added afterwards.

``BF16`` is the largest relative error of one rounding to bf16 (2^-8).
"""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

BF16 = 2.0 ** -8


def _rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-30)).item()


def _segments(kind, b, s):
    at = torch.arange(s).repeat(b, 1)
    if kind == "one":
        seg = torch.ones(b, s)
    elif kind == "short":                       # a tile sees two or three 64-row blocks a head
        seg = at // 40 + 1
    elif kind == "uneven":                      # tiles with one, with several and with the most items, odd numbers of blocks
        seg = (at >= 70).int() + (at >= 200).int() + (at >= 3 * s // 4 - 9).int() + 1
    else:                                       # some tiles are seen by nobody
        seg = ((at >= 300) & (at < s - 200)).int()
    return seg.int().cuda()


@pytest.mark.parametrize("kind", ["one", "short", "uneven", "padded"])
@pytest.mark.parametrize("b,s,hq,hkv,d", [(1, 1152, 14, 2, 128), (1, 2048, 4, 1, 64), (2, 640, 12, 2, 128), (1, 1024, 2, 1, 64)])
def test_key_tiles_in_parts(cuda_lib, monkeypatch, kind, b, s, hq, hkv, d):
    from causal_trainer_dev_b200.ops import attention as A

    lib = cuda_lib.lib()
    wanted = lib.ctb_attn_bwd_workspace(b, s, s, hq, hkv, d)
    assert wanted >= 2 * b * hkv * s * d * 2 * 4 and wanted % (b * hkv * s * d * 2 * 4) == 0
    gen = torch.Generator(device="cuda").manual_seed(1)
    qkv = torch.randn(b, s, hq + 2 * hkv, d, generator=gen, device="cuda").bfloat16()
    q, k, v = qkv[:, :, :hq], qkv[:, :, hq:hq + hkv], qkv[:, :, hq + hkv:]
    do = torch.randn(b, s, hq, d, generator=gen, device="cuda").bfloat16()
    seg = _segments(kind, b, s)
    meta = A.build_attention_meta(seg)
    o, lse = A.flash_attention_forward(q, k, v, meta)

    def backward(**more):
        packed = torch.full_like(qkv, 7.0)          # strided outputs, written everywhere
        outs = dict(dq=packed[:, :, :hq], dk=packed[:, :, hq:hq + hkv], dv=packed[:, :, hq + hkv:])
        outs.update(more)
        got = A.flash_attention_backward(q, k, v, o, do, lse, meta, **outs)
        assert cuda_lib.device_status() == (0, 0, 0, 0)
        return [t.clone() for t in got]

    first = backward()
    assert all(torch.equal(x, y) for x, y in zip(first, backward()))
    over_dout = do.clone()                          # dQ in the place of dO: dK / dV are a launch of their own
    alias = A.flash_attention_backward(q, k, v, o, over_dout, lse, meta, dq=over_dout)
    assert all(torch.equal(x, y) for x, y in zip(first, alias))
    # queries [s / 2, s): what sequence parallelism asks of a rank (its key tiles have other numbers of items)
    half = s // 256 * 128
    held = [t[:, half:].contiguous() for t in (q, o, do)] + [lse[:, :, half:].contiguous()]
    part = A.flash_attention_backward(held[0], k, v, *held[1:], meta, q_offset=half)
    monkeypatch.setattr(lib, "ctb_attn_bwd_workspace", lambda *a: 0)
    whole = backward()
    whole_part = A.flash_attention_backward(held[0], k, v, *held[1:], meta, q_offset=half)
    assert torch.equal(first[0], whole[0]) and torch.equal(part[0], whole_part[0])
    for got, want in ((first[1], whole[1]), (first[2], whole[2]), (part[1], whole_part[1]), (part[2], whole_part[2])):
        assert _rel(got, want) < 2 * BF16           # two roundings to bf16 of sums in another order
        if kind == "short" and hq == 2 * hkv:       # at most three blocks a head: less than two items' work
            assert torch.equal(got, want)
    group, i = hq // hkv, b - 1
    qd, kd, vd = (t[i].double().requires_grad_() for t in (q, k, v))
    score = torch.einsum("qhd,khd->hqk", qd, kd.repeat_interleave(group, 1)) / math.sqrt(d)
    see = A.visibility_mask(seg[i:i + 1])[0]
    p = torch.where(see.any(-1)[None, :, None], score.masked_fill(~see, -math.inf), torch.zeros_like(score)).softmax(-1) * see
    torch.einsum("hqk,khd->qhd", p, vd.repeat_interleave(group, 1)).backward(do[i].double())
    for got, want in zip(first, (qd.grad, kd.grad, vd.grad)):
        assert _rel(got[i], want) < 3 * BF16


@pytest.mark.parametrize("b,s,hq,hkv,d,docs", [(2, 2048, 14, 2, 128, 128), (1, 4096, 8, 2, 128, 128), (1, 4096, 8, 2, 64, 64)])
def test_tiles_of_short_documents_stay_whole(cuda_lib, monkeypatch, b, s, hq, hkv, d, docs):
    """Rows that would be cut as one document, but whose documents leave no part the work it has to have at least: the bits of
    the uncut call."""
    from causal_trainer_dev_b200.ops import attention as A

    assert cuda_lib.lib().ctb_attn_bwd_workspace(b, s, s, hq, hkv, d) > 0
    gen = torch.Generator(device="cuda").manual_seed(4)
    q, do = (torch.randn(b, s, hq, d, generator=gen, device="cuda").bfloat16() for _ in range(2))
    k, v = (torch.randn(b, s, hkv, d, generator=gen, device="cuda").bfloat16() for _ in range(2))
    meta = A.build_attention_meta((torch.arange(s, device="cuda") // docs + 1).int().repeat(b, 1))
    o, lse = A.flash_attention_forward(q, k, v, meta)
    got = A.flash_attention_backward(q, k, v, o, do, lse, meta)
    monkeypatch.setattr(cuda_lib.lib(), "ctb_attn_bwd_workspace", lambda *a: 0)
    want = A.flash_attention_backward(q, k, v, o, do, lse, meta)
    assert all(torch.equal(x, y) for x, y in zip(got, want))
    assert cuda_lib.device_status() == (0, 0, 0, 0)


def test_no_memory_for_the_parts(cuda_lib, monkeypatch):
    """An allocation that fails: the call is uncut, with the bits of the uncut call."""
    from causal_trainer_dev_b200.ops import attention as A

    b, s, hq, hkv, d = 1, 2048, 14, 2, 128
    wanted = cuda_lib.lib().ctb_attn_bwd_workspace(b, s, s, hq, hkv, d)
    assert wanted > 16 << 20
    gen = torch.Generator(device="cuda").manual_seed(5)
    q, do = (torch.randn(b, s, hq, d, generator=gen, device="cuda").bfloat16() for _ in range(2))
    k, v = (torch.randn(b, s, hkv, d, generator=gen, device="cuda").bfloat16() for _ in range(2))
    meta = A.build_attention_meta(torch.ones(b, s, dtype=torch.int32, device="cuda"))
    o, lse = A.flash_attention_forward(q, k, v, meta)
    cut, got = ([torch.empty_like(x) for x in (q, k, v)] for _ in range(2))
    A.flash_attention_backward(q, k, v, o, do, lse, meta, dq=cut[0], dk=cut[1], dv=cut[2])
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.empty_cache()
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (6 << 20)) / total)
    before = cuda_lib.launch_count()
    try:
        held = []
        with pytest.raises(torch.cuda.OutOfMemoryError):
            while True:                                          # what the allocator has left in large pieces
                held.append(torch.empty(16 << 20, dtype=torch.uint8, device="cuda"))
        A.flash_attention_backward(q, k, v, o, do, lse, meta, dq=got[0], dk=got[1], dv=got[2])
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
        del held
    assert cuda_lib.launch_count() == before + 2                # no kernel for the sums
    monkeypatch.setattr(cuda_lib.lib(), "ctb_attn_bwd_workspace", lambda *a: 0)
    want = A.flash_attention_backward(q, k, v, o, do, lse, meta)
    assert all(torch.equal(x, y) for x, y in zip(got, want)) and not torch.equal(got[1], cut[1])
    assert cuda_lib.device_status() == (0, 0, 0, 0)


@pytest.mark.parametrize("b,s,hq,hkv,d", [(1, 1152, 14, 2, 128), (2, 1024, 12, 2, 128), (1, 2048, 4, 1, 64)])
def test_parts_of_tiles_with_image_spans(cuda_lib, monkeypatch, b, s, hq, hkv, d):
    """Spans whose tokens see each other (attention_end), across tile borders and in two documents."""
    from causal_trainer_dev_b200.ops import attention as A

    assert cuda_lib.lib().ctb_attn_bwd_workspace(b, s, s, hq, hkv, d) > 0
    gen = torch.Generator(device="cuda").manual_seed(6)
    q, do = (torch.randn(b, s, hq, d, generator=gen, device="cuda").bfloat16() for _ in range(2))
    k, v = (torch.randn(b, s, hkv, d, generator=gen, device="cuda").bfloat16() for _ in range(2))
    seg = (torch.arange(s).repeat(b, 1) >= s - 200).int() + 1
    end = torch.arange(s, dtype=torch.int32).repeat(b, 1)
    for first, last in ((100, 355), (500, 755), (760, 790), (s - 190, s - 1)):
        end[:, first:last + 1] = last
    seg, end = seg.cuda(), end.cuda()
    meta = A.build_attention_meta(seg, end)
    o, lse = A.flash_attention_forward(q, k, v, meta)
    got = A.flash_attention_backward(q, k, v, o, do, lse, meta)
    assert all(torch.equal(x, y) for x, y in zip(got, A.flash_attention_backward(q, k, v, o, do, lse, meta)))
    monkeypatch.setattr(cuda_lib.lib(), "ctb_attn_bwd_workspace", lambda *a: 0)
    whole = A.flash_attention_backward(q, k, v, o, do, lse, meta)
    assert torch.equal(got[0], whole[0]) and not torch.equal(got[1], whole[1])
    group, i = hq // hkv, b - 1
    qd, kd, vd = (t[i].double().requires_grad_() for t in (q, k, v))
    see = A.visibility_mask(seg[i:i + 1], end[i:i + 1])[0]
    score = torch.einsum("qhd,khd->hqk", qd, kd.repeat_interleave(group, 1)) / math.sqrt(d)
    p = score.masked_fill(~see, -math.inf).softmax(-1)
    torch.einsum("hqk,khd->qhd", p, vd.repeat_interleave(group, 1)).backward(do[i].double())
    for x, y, want in zip(got, whole, (qd.grad, kd.grad, vd.grad)):
        assert _rel(x[i], want) < 3 * BF16 and _rel(x[i], want) < 1.02 * _rel(y[i], want)      # no further off than uncut
    assert cuda_lib.device_status() == (0, 0, 0, 0)
