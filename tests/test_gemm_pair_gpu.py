"""The two-CTA products: every form that the choice by size may take, at the ends of tiles, slices and bands, against 64
bits; and the loss epilogues on it against the one-CTA kernel.

``BF16`` is the largest relative error of one rounding to bf16 (2^-8).
"""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

BF16 = 2.0 ** -8


def _rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-30)).item()


def _bf16(*shape, seed=0, scale=1.0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, generator=gen, device="cuda") * scale).bfloat16()


def _pad(x):
    return -(-x // 8) * 8


@pytest.mark.parametrize("tm", [1, 2])
@pytest.mark.parametrize("m,n,k,whole,slices,band", [
    (1, 8, 8, 1, 1, 8), (257, 257, 520, -1, 1, 16), (130, 270, 1000, 0, 3, 8), (513, 131, 72, -1, 1, 1),
    (1100, 700, 520, 1, 8, 2), (300, 1300, 4104, 0, 5, 8), (700, 300, 264, 1, 2, 1)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
def test_every_form(cuda_lib, tm, m, n, k, whole, slices, band, a_mn, b_mn):
    tiles = -(-m // (256 * tm)) * -(-n // 256)
    whole = tiles if whole < 0 else min(whole, tiles)
    a = _bf16(k, _pad(m), seed=1)[:, :m] if a_mn else _bf16(m, _pad(k), seed=1)[:, :k]
    b = _bf16(k, _pad(n), seed=2)[:, :n] if b_mn else _bf16(n, _pad(k), seed=2)[:, :k]
    want = (a.double().t() if a_mn else a.double()) @ (b.double() if b_mn else b.double().t())
    bias, p, ln = _bf16(n, seed=3), cuda_lib.ptr, ctypes.c_long
    size = (tiles - whole) * slices * 256 * tm * 256 * 4
    work = torch.full((size + 256,), 255, dtype=torch.uint8, device="cuda")

    def run(dtype, alpha, bias, accumulate=0, start=7.0, work_bytes=size):
        out = torch.full((m + 3, _pad(n) + 8), start, dtype=dtype, device="cuda")
        code = cuda_lib.lib().ctb_gemm_pair(
            p(a), p(b), p(out), m, n, k, ln(a.stride(0)), ln(b.stride(0)), ln(out.stride(0)), int(a_mn), int(b_mn),
            int(dtype == torch.float32), accumulate, ctypes.c_float(alpha), p(bias), tm, whole, slices, band, p(work),
            ln(work_bytes), cuda_lib.stream_ptr())
        if code:
            return None
        # the frame is left alone, but for the rest of a row's last 16 bytes (TMA stores whole ones; the choice by size takes
        # no such rows)
        assert torch.all(out[:, _pad(n):] == start) and torch.all(out[m:] == start)
        assert torch.all(work[size:] == 255)
        return out[:m, :n]

    assert _rel(run(torch.bfloat16, 1.0, None), want) < BF16
    assert _rel(run(torch.bfloat16, 0.5, bias), (want + bias.double()) * 0.5) < BF16
    assert _rel(run(torch.float32, 0.5, None), want * 0.5) < 1e-5                    # fp32 sums of 4104 products
    if whole == tiles:
        assert _rel(run(torch.float32, 0.5, None, accumulate=1, start=2.0), want * 0.5 + 2) < 1e-5
    else:
        assert run(torch.float32, 1.0, None, accumulate=1) is None                   # refused: split tiles are stored
        assert run(torch.float32, 1.0, None, work_bytes=size - 4) is None            # and need their whole workspace
    assert cuda_lib.device_status() == (0, 0, 0, 0)


@pytest.mark.parametrize("rows,vocab,d,tm", [
    (1000, 32000, 1536, 1), (4000, 5000, 256, 1), (1, 2520, 976, 1),
    (644, 6216, 584, 2), (894, 7376, 896, 2), (452, 12400, 1328, 2), (288, 13232, 616, 2), (2077, 2064, 608, 2),
    (300, 20000, 520, None)])                     # None: the one-CTA kernel by size, too
def test_loss_epilogues_on_two_ctas(cuda_lib, rows, vocab, d, tm):
    from causal_trainer_dev_b200.ops import cross_entropy as ce

    form = (ctypes.c_int * 4)()
    for gradients in (0, 1):
        taken = cuda_lib.lib().ctb_ce_pair_choice(rows, vocab, d, gradients, form)
        assert (form[0] if taken else None) == tm
    hidden, head = _bf16(rows, d, seed=1), _bf16(vocab, d, seed=2, scale=0.05)
    gen = torch.Generator(device="cuda").manual_seed(3)
    targets = torch.randint(0, vocab, (rows,), generator=gen, device="cuda")
    weights = (torch.rand(rows, generator=gen, device="cuda") < 0.7).float()
    results = []
    before = cuda_lib.lib().ctb_gemm_set_pair(-1)
    try:
        for mode in (-1, 0):
            cuda_lib.lib().ctb_gemm_set_pair(mode)
            nll, total, lse, coef = ce.cut_ce_forward(hidden, head, targets, weights, 1e-3)
            results.append((nll, total, lse, coef, *ce.cut_ce_backward(hidden, head, targets, lse, coef)))
    finally:
        cuda_lib.lib().ctb_gemm_set_pair(before)
    # one order of the sums within a tile: statistics within fp32 rounding, gradients within one of bf16
    for got, want, limit in zip(*results, (1e-6, 0, 1e-6, 0, BF16, BF16)):
        assert _rel(got, want) <= limit
    logits = hidden.double() @ head.double().t()
    lse = torch.logsumexp(logits, -1)
    assert _rel(results[0][2], lse) < 1e-6
    g = (logits - lse[:, None]).exp()
    g[torch.arange(rows, device="cuda"), targets] -= 1
    g *= (weights.double() * 1e-3)[:, None]
    assert _rel(results[0][4], g @ head.double()) < 2 * BF16 and _rel(results[0][5], g.t() @ hidden.double()) < 2 * BF16
    assert cuda_lib.device_status() == (0, 0, 0, 0)
