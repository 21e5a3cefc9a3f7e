"""Target ids of both widths, contiguous or not, inside and outside the vocabulary, and both kinds of gradient scale: the loss
functions read ids in place and leave out the rows that have none."""
import pytest
import torch

pytestmark = pytest.mark.gpu

BF16 = 2.0 ** -8


@pytest.mark.parametrize("rows,vocab,d,chunk", [(1, 256, 256, 4096), (333, 1000, 512, 96), (70, 4104, 512, 4096), (9000, 520, 256, 4096)])
def test_forms_of_targets_and_scales(cuda_lib, rows, vocab, d, chunk):
    from causal_trainer_dev_b200.ops import cross_entropy as CE

    gen = torch.Generator(device="cuda").manual_seed(rows)
    h = torch.randn(rows, d, generator=gen, device="cuda").bfloat16()
    w = (torch.randn(vocab, d, generator=gen, device="cuda") * 0.05).bfloat16()
    t = torch.randint(0, vocab, (rows,), generator=gen, device="cuda")
    t[rows // 2::7] = -1                                     # no target: the row's loss is its log-sum-exp
    t[0] = vocab - 1
    weights = torch.rand(rows, generator=gen, device="cuda")
    weights[rows // 3::5] = 0.0
    weights[0] = 0.5
    scale = torch.tensor([0.37], device="cuda")
    wide = torch.stack((t, t + 1), dim=1)[:, 0]              # not contiguous
    forms = [(t, scale), (t.int(), scale), (wide, scale), (t, 0.37), (t, scale.double())]
    results = []
    for targets, factor in forms:
        nll, total, lse, coef = CE.cut_ce_forward(h, w, targets, weights, factor)
        dh, dw = CE.cut_ce_backward(h, w, targets, lse, coef, chunk_rows=chunk)
        both = CE.cut_ce_forward_backward(h, w, targets, weights, factor, chunk_rows=chunk)
        results.append((nll, total, lse, coef, dh, dw, *both))
    for other in results[1:]:
        assert all(torch.equal(x, y) for x, y in zip(results[0], other))
    nll, total, lse, coef, dh, dw, nll2, total2, dh2, dw2 = results[0]
    assert torch.equal(total, total2) and torch.equal(dh, dh2)
    logits = h.double() @ w.double().T
    exact = torch.logsumexp(logits, 1)
    picked = torch.where(t >= 0, logits.gather(1, t.clamp_min(0)[:, None])[:, 0], torch.zeros_like(exact))
    want = ((exact - picked) * weights.double()).sum()
    # fp32 sums of bf16 products: 1e-5 of the terms' size each
    assert abs(float(nll) - float(want)) < 1e-5 * float(((exact.abs() + picked.abs()) * weights.double()).sum())
    assert abs(float(nll2) - float(want)) < 1e-5 * float(((exact.abs() + picked.abs()) * weights.double()).sum())
    assert abs(float(total) - float(weights.double().sum())) < 1e-5 * float(weights.double().sum())
    g = torch.softmax(logits, 1)
    g[torch.arange(rows, device="cuda")[t >= 0], t[t >= 0]] -= 1
    g *= (weights.double() * 0.37)[:, None]
    for got, ref in ((dh, g @ w.double()), (dw, g.T @ h.double()), (dw2, g.T @ h.double())):
        assert ((got.double() - ref).norm() / ref.norm()).item() < 2 * BF16      # g and the results are rounded
