"""Attention kernels with more work items than SMs: CTAs that take over items which have not started, with and
without work, in the middle of others of another length or kind.

Compared with a 64-bit PyTorch statement of the same operation.  ``BF16`` is the largest relative error of one
rounding to bf16 (2^-8): P and dS are rounded before the products and the results once more.
"""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

BF16 = 2.0 ** -8


def _rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-30)).item()


def _runs(b, s, padding):
    """Documents of very different lengths; ``padding`` rows of every batch see nothing, so some items have no work."""
    seg = torch.zeros(b, s, dtype=torch.int32)
    for i in range(b):
        at, n, label = padding * (i % 2), 37 + 11 * i, 1
        while at < s - padding:
            seg[i, at:min(at + n, s - padding)] = label
            at, n, label = at + n, n * 2, label + 1
    return seg.cuda()


@pytest.mark.parametrize("d,hq,hkv", [(128, 8, 2), (64, 12, 2), (128, 6, 6)])
@pytest.mark.parametrize("b,s,padding", [(6, 896, 0), (4, 1152, 300), (3, 1408, 640)])
def test_more_work_items_than_sms(cuda_lib, d, hq, hkv, b, s, padding):
    from causal_trainer_dev_b200.ops import attention as A

    assert b * hq * (-(-s // 256)) > 90 and b * s // 128 * (hq + hkv) > 2 * 148
    gen = torch.Generator(device="cuda").manual_seed(1)
    q, k, v, do = (torch.randn(b, s, h, d, generator=gen, device="cuda").bfloat16() for h in (hq, hkv, hkv, hq))
    seg = _runs(b, s, padding)
    meta = A.build_attention_meta(seg)
    first = None
    for _ in range(3):
        out = torch.full_like(q, 7.0)
        o, lse = A.flash_attention_forward(q, k, v, meta, out=out)
        grads = A.flash_attention_backward(q, k, v, o, do, lse, meta)
        assert cuda_lib.device_status() == (0, 0, 0, 0)
        if first is None:
            first = (o, lse, *grads)
        assert all(torch.equal(x, y) for x, y in zip(first, (o, lse, *grads)))      # whatever CTA an item ran in
    group = hq // hkv
    for i in range(b):                                                              # (a batch row at a time: memory)
        qd, kd, vd = (t[i].double().requires_grad_() for t in (q, k, v))
        score = torch.einsum("qhd,khd->hqk", qd, kd.repeat_interleave(group, 1)) / math.sqrt(d)
        see = A.visibility_mask(seg[i:i + 1])[0]
        p = torch.where(see.any(-1)[None, :, None], score.masked_fill(~see, -math.inf), torch.zeros_like(score)).softmax(-1) * see
        ref = torch.einsum("hqk,khd->qhd", p, vd.repeat_interleave(group, 1))
        ref.backward(do[i].double())
        for got, want in zip((first[0], *first[2:]), (ref, qd.grad, kd.grad, vd.grad)):
            assert _rel(got[i], want) < 3 * BF16
        assert bool((first[0][i][seg[i] == 0] == 0).all())
