"""The head's forward and backward in one, with a chunk's logits kept in fp32, against the two calls that compute them
twice: the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,vocab,d,chunk", [(1, 8, 1024, 4096), (333, 4104, 1024, 128), (700, 2048, 1032, 256), (260, 2056, 1024, 4096),
                                                (600, 20008, 1536, 512), (129, 4104, 512, 64), (129, 4104, 504, 64),
                                                (894, 7376, 896, 4096), (904, 12400, 1328, 452)])      # two CTAs, 512 rows
@pytest.mark.parametrize("on_device,accumulate", [(False, False), (True, True)])
def test_one_call_is_the_two(cuda_lib, rows, vocab, d, chunk, on_device, accumulate):
    from causal_trainer_dev_b200.ops import cross_entropy as ce

    gen = torch.Generator(device="cuda").manual_seed(rows)
    hidden = torch.randn(rows, d, generator=gen, device="cuda").bfloat16()
    head = (torch.randn(vocab, d, generator=gen, device="cuda") * 0.05).bfloat16()
    targets = torch.randint(0, vocab, (rows,), generator=gen, device="cuda")
    weights = (torch.rand(rows, generator=gen, device="cuda") < 0.6).float() * 1.5
    scale = torch.tensor(1e-2, device="cuda") if on_device else 1e-2
    start = torch.randn(vocab, d, generator=gen, device="cuda")
    one, two = start.clone(), start.clone()
    nll, total, lse, coef = ce.cut_ce_forward(hidden, head, targets, weights, scale)
    dh, _ = ce.cut_ce_backward(hidden, head, targets, lse, coef, chunk_rows=chunk, dhead_out=two, dhead_accumulate=accumulate)
    nll1, total1, dh1, dhead1 = ce.cut_ce_forward_backward(hidden, head, targets, weights, scale, chunk_rows=chunk,
                                                           dhead_out=one, dhead_accumulate=accumulate)
    assert dhead1 is one
    for a, b in ((nll1, nll), (total1, total), (dh1, dh), (one, two)):
        assert torch.equal(a, b)
    assert ce.cut_ce_forward_backward(hidden, head, targets, weights, scale, chunk_rows=chunk, need_dhead=False)[3] is None
    assert cuda_lib.device_status() == (0, 0, 0, 0)


def test_a_vocabulary_that_the_two_refuse(cuda_lib):
    from causal_trainer_dev_b200.ops import cross_entropy as ce

    hidden, head = (torch.zeros(n, 1024, dtype=torch.bfloat16, device="cuda") for n in (64, 1001))
    with pytest.raises(cuda_lib.KernelError, match="16 bytes"):
        ce.cut_ce_forward_backward(hidden, head, torch.zeros(64, dtype=torch.long, device="cuda"), torch.ones(64, device="cuda"))


@pytest.mark.parametrize("how", ["no memory", "not wanted"])
def test_without_memory_for_the_logits(cuda_lib, monkeypatch, how):
    """The slab that is refused, or not asked for: the two calls, and no slab of four bytes a logit."""
    from causal_trainer_dev_b200.ops import cross_entropy as ce

    gen = torch.Generator(device="cuda").manual_seed(1)
    hidden = torch.randn(300, 1024, generator=gen, device="cuda").bfloat16()
    head = (torch.randn(4104, 1024, generator=gen, device="cuda") * 0.05).bfloat16()
    targets = torch.randint(0, 4104, (300,), generator=gen, device="cuda")
    weights = torch.ones(300, device="cuda")
    want = ce.cut_ce_forward_backward(hidden, head, targets, weights, 1e-2, chunk_rows=128)
    empty, asked = torch.empty, []

    def refuse(*args, **kw):
        shape = args[0] if len(args) == 1 and not isinstance(args[0], int) else args
        if tuple(shape) == (128, 4104) and kw.get("dtype") == torch.float32:
            asked.append(shape)
            raise torch.cuda.OutOfMemoryError("refused by the test")
        return empty(*args, **kw)

    monkeypatch.setattr(torch, "empty", refuse)
    got = ce.cut_ce_forward_backward(hidden, head, targets, weights, 1e-2, chunk_rows=128, keep_logits=how == "no memory")
    assert len(asked) == (how == "no memory")
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    assert cuda_lib.device_status() == (0, 0, 0, 0)
