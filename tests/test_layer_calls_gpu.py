"""Layers issued as one library call per direction, and next-token targets from one kernel, against the same schedule
launch by launch from Python and against the tensor formulation: the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _batch(rows, seq, vocab, gen):
    ids = torch.randint(3, vocab, (rows, seq), generator=gen, device="cuda")
    mask = torch.ones_like(ids)
    mask[-1, seq - 77:] = 0
    seg = torch.ones_like(ids)
    seg[:, seq // 3:] = 2
    return dict(input_ids=ids, attention_mask=mask, segment_ids=seg)


@pytest.mark.parametrize("options", [{}, {"remat": "full"}, {"remat": "full", "remat_group_size": 2}, {"train_norm": False}])
@pytest.mark.parametrize("bias,style,grad_dtype", [(False, "gpt-neox", torch.bfloat16), (True, "gpt-j", torch.float32)])
def test_a_pass_gives_the_same_bits_either_way(cuda_lib, monkeypatch, options, bias, style, grad_dtype):
    from causal_trainer_dev_b200.models.config import preset
    from causal_trainer_dev_b200.models.params import ModelParams
    from causal_trainer_dev_b200.training import engine as E

    cfg = preset("tiny", num_hidden_layers=3, vocab_size=1000, attention_bias=bias, rope_style=style)
    gen = torch.Generator(device="cuda").manual_seed(3)
    batches = [_batch(2, 384, 1000, gen) for _ in range(2)]
    results = []
    for limit in (E.LAYER_CALL_BYTES, 0):
        monkeypatch.setattr(E, "LAYER_CALL_BYTES", limit)
        params = ModelParams.init_random(cfg, seed=1).to("cuda")
        engine = E.LayerwiseEngine(cfg, E.LocalProvider(params, grad_dtype), E.EngineOptions(**options))
        sums = [engine(b, 1e-2, first=i == 0) for i, b in enumerate(batches)]
        calls = engine._layer_calls(engine._context(batches[0]), torch.empty(768, cfg.hidden_size, dtype=torch.bfloat16, device="cuda"))
        assert (calls is not None) == (limit > 0)
        results.append([x for s in sums for x in s] + [u.grad for u in params.units.values()])
    for a, b in zip(*results):
        assert torch.equal(a, b)
    assert all(bool(torch.isfinite(g.float()).all()) for g in results[0][4:])
    assert cuda_lib.device_status() == (0, 0, 0, 0)


@pytest.mark.parametrize("id_dtype", [torch.int64, torch.int32])
@pytest.mark.parametrize("mask_dtype", [torch.int64, torch.int32, torch.bool, None])
@pytest.mark.parametrize("labels", [True, False])
@pytest.mark.parametrize("loss", [True, False])
def test_targets_from_one_kernel(cuda_lib, id_dtype, mask_dtype, labels, loss):
    from causal_trainer_dev_b200.training import losses

    gen = torch.Generator(device="cuda").manual_seed(5)
    b, s = 3, 333
    ids = torch.randint(0, 50, (b, s), generator=gen, device="cuda").to(id_dtype)
    ids[0, 7] = -100
    batch = {"input_ids": ids}
    if mask_dtype is not None:
        mask = torch.rand(b, s, generator=gen, device="cuda") < 0.8
        batch["attention_mask"] = mask.to(mask_dtype)
        if mask_dtype == torch.int64:
            batch["attention_mask"][1, 5:9] = 2                   # only 1 is valid
    if labels:
        batch["segment_ids"] = torch.randint(0, 2, (b, s), generator=gen, device="cuda")
    if loss:
        batch["loss_weights"] = torch.randn(b, s, generator=gen, device="cuda")
    want_t, want_w = losses.aligned_targets_and_weights(batch)
    before = cuda_lib.launch_count()
    got_t, got_w = losses.device_targets_and_weights(batch)
    assert cuda_lib.launch_count() == before + 1 and got_t.dtype == torch.int32
    assert torch.equal(got_t.long(), want_t) and torch.equal(got_w, want_w)
    batch["prediction_targets"], batch["prediction_weights"] = ids.long().abs(), torch.ones(b, s, device="cuda")
    assert torch.equal(losses.device_targets_and_weights(batch)[0], losses.aligned_targets_and_weights(batch)[0])


def test_a_switch_turned_between_the_passes(cuda_lib):
    """Blocks are sized for the products' kernels of the moment: a pass with the two-CTA kernel off, one with it, and the
    other way round, each the same bits as a pass of its own."""
    from causal_trainer_dev_b200.models.config import preset
    from causal_trainer_dev_b200.models.params import ModelParams
    from causal_trainer_dev_b200.training import engine as E

    cfg = preset("qwen2.5-1.5b-image", num_hidden_layers=1, vocab_size=1000, pad_token_id=0, eos_token_id=2)
    batch = _batch(1, 384, 1000, torch.Generator(device="cuda").manual_seed(3))
    set_pair = cuda_lib.lib().ctb_gemm_set_pair
    before = set_pair(-1)
    try:
        seen = {}
        for mode in (0, -1, 0, -1):
            set_pair(mode)
            params = ModelParams.init_random(cfg, seed=1).to("cuda")
            engine = E.LayerwiseEngine(cfg, E.LocalProvider(params, torch.bfloat16))
            sums = engine(batch, 1e-2, first=True)
            assert engine._layer_calls(engine._context(batch), torch.empty(384, cfg.hidden_size, dtype=torch.bfloat16, device="cuda"))
            got = [*sums, *(u.grad for u in params.units.values())]
            assert all(torch.equal(a, b) for a, b in zip(seen.setdefault(mode, got), got))
    finally:
        set_pair(before)
    assert cuda_lib.device_status() == (0, 0, 0, 0)


def test_a_pass_without_room_for_partial_sums(cuda_lib, monkeypatch):
    """A backward block that cannot be had is asked for again without the partial sums of dK / dV: the bits of the schedule from
    Python without them, and two roundings of the results with them."""
    from causal_trainer_dev_b200.models.config import preset
    from causal_trainer_dev_b200.models.params import ModelParams
    from causal_trainer_dev_b200.training import engine as E

    cfg = preset("tiny", num_hidden_layers=2, vocab_size=1000)
    lib, heads = cuda_lib.lib(), (cfg.num_attention_heads, cfg.num_key_value_heads, cfg.head_dim)
    assert lib.ctb_attn_bwd_workspace(1, 1024, 1024, *heads) > 0
    gen = torch.Generator(device="cuda").manual_seed(3)
    ids = torch.randint(3, 1000, (1, 1024), generator=gen, device="cuda")
    batch = dict(input_ids=ids, attention_mask=torch.ones_like(ids), segment_ids=torch.ones_like(ids))
    seen, real = [], torch.empty

    def run(refuse):
        params = ModelParams.init_random(cfg, seed=1).to("cuda")
        engine = E.LayerwiseEngine(cfg, E.LocalProvider(params, torch.bfloat16))
        calls = engine._layer_calls(engine._context(batch), real(1024, cfg.hidden_size, dtype=torch.bfloat16, device="cuda"))

        def empty(*size, **how):
            if size == (calls._backward,):
                seen.append(size)
                raise torch.cuda.OutOfMemoryError("no memory for the block")
            return real(*size, **how)

        with monkeypatch.context() as m:
            if refuse:
                m.setattr(torch, "empty", empty)
            sums = engine(batch, 1e-2, first=True)
        return [*sums, *(u.grad for u in params.units.values())], calls

    with_sums, calls = run(False)
    assert calls.backward_launches == 23 and not seen
    without, _ = run(True)
    assert len(seen) == 1                                   # the second layer asks for what there is
    monkeypatch.setattr(E, "LAYER_CALL_BYTES", 0)
    monkeypatch.setattr(lib, "ctb_attn_bwd_workspace", lambda *a: 0)
    python, calls = run(False)
    assert calls is None and all(torch.equal(a, b) for a, b in zip(without, python))
    assert not all(torch.equal(a, b) for a, b in zip(without, with_sums))
    for a, b in zip(without, with_sums):
        assert ((a.double() - b.double()).norm() <= 2.0 ** -6 * b.double().norm()).item()      # bf16 roundings of two layers
    assert cuda_lib.device_status() == (0, 0, 0, 0)
