"""The work that users of this trainer have it do, as cases that can be timed and compared.

Most cases are one layer-sized piece of a training step, forward and backward, called through the
functions of ``causal_trainer_dev_b200.ops`` with the layouts that the engine and user programs hand
in (q, k and v as views of one packed projection output, gradients into views of one packed buffer).
Two are a whole engine pass over a micro-batch.  Shapes are those of ``models.config.PRESETS`` (at one
GPU or as one tensor-parallel rank of four sees them), of the tests, or generic; rows come from
``data.synthetic``, the corpora that ``bench.py`` trains on.
"""
import math

import numpy as np
import torch

from causal_trainer_dev_b200.data import synthetic
from causal_trainer_dev_b200.models.config import preset
from causal_trainer_dev_b200.models.params import ModelParams
from causal_trainer_dev_b200.ops import attention, cross_entropy, elementwise, gemm, moba
from causal_trainer_dev_b200.training.engine import LayerwiseEngine, LocalProvider

BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64


# ---------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest attention call: two short rows of the tests' tiny shape, all launches and latency
        dict(name="attention_tiny", kind="attention", rows=2, seq=256, heads=4, kv_heads=2, dim=64, docs="packed"),
        # one layer of the default benchmark: an 8B micro-batch of packed documents (median 600 tokens)
        dict(name="attention_packed", kind="attention", rows=4, seq=4096, heads=32, kv_heads=8, dim=128, docs="packed"),
        # long-context training on one document per row, as one of four tensor-parallel ranks sees it
        dict(name="attention_document", kind="attention", rows=1, seq=32768, heads=8, kv_heads=2, dim=128, docs="one"),
        # mixed autoregressive + image-grid rows of the 1.5B shape (block-local bidirectional spans)
        dict(name="attention_images", kind="attention", rows=8, seq=4096, heads=12, kv_heads=2, dim=128, docs="images"),
        # block-sparse layer of the 32k configuration: one document, block 4096, top-3 + current
        dict(name="moba_32k", kind="moba", rows=1, seq=32768, heads=32, kv_heads=8, dim=128, docs="one", block=4096,
             top_k=4),
        # norm + gated MLP of an 8B layer on a full micro-batch of 16384 tokens: the largest GEMMs
        dict(name="mlp_8b", kind="mlp", tokens=16384, hidden=4096, inner=14336),
        # the same layer piece of the 1.5B shape on a ragged number of rows (a short last batch)
        dict(name="mlp_ragged", kind="mlp", tokens=1000, hidden=1536, inner=8960),
        # language-model head and loss of an 8B micro-batch chunk, every row supervised
        dict(name="head_8b", kind="head", rows=4096, hidden=4096, vocab=128256, weighted=1.0),
        # the head on a few supervised rows (assistant-only fine-tuning after row compaction), odd sizes
        dict(name="head_few_rows", kind="head", rows=333, hidden=1536, vocab=32000, weighted=0.9),
        # clip norm and AdamW over one 8B layer's flat parameter buffer, as the optimizer sweeps units
        dict(name="optimizer_layer", kind="optimizer", count=218112000, accumulate=True),
        # a whole engine pass of the tiny configuration (what smoke tests and small experiments run)
        dict(name="step_tiny", kind="step", model="tiny", layers=2, rows=2, seq=256, docs="packed"),
        # a whole engine pass of the 1.5B image shape cut to two layers: biases, rotary embedding, row
        # compaction, embedding gradients, a large vocabulary
        dict(name="step_images", kind="step", model="qwen2.5-1.5b-image", layers=2, rows=2, seq=4096, docs="images"),
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["attention", "attention", "attention", "moba", "mlp", "mlp", "head", "optimizer", "step"])
    if kind in ("attention", "moba"):
        heads, kv_heads, dim = rng.choice([(32, 8, 128), (8, 2, 128), (12, 2, 128), (28, 4, 128), (14, 2, 128), (4, 2, 64),
                                           (16, 4, 64)])
    if kind == "attention":
        docs = rng.choice(["packed", "packed", "one", "several", "images"])
        seq = 128 * _spread(rng, 16 if docs == "images" else 1, 256 if docs in ("one", "several") and heads <= 8 else 64)
        return dict(kind=kind, rows=max(1, min(_spread(rng, 1, 24), 16384 // seq)), seq=seq, heads=heads,
                    kv_heads=kv_heads, dim=dim, docs=docs)
    if kind == "moba":
        return dict(kind=kind, rows=1, seq=128 * _spread(rng, 32, 200), heads=heads, kv_heads=kv_heads, dim=dim,
                    docs=rng.choice(["one", "several"]), block=rng.choice([512, 1024, 2048]), top_k=rng.randint(2, 4))
    if kind == "mlp":
        hidden, inner = rng.choice([(4096, 14336), (1536, 8960), (3584, 18944), (256, 688), (4096, 3584)])
        return dict(kind=kind, tokens=_spread(rng, 64, 12000), hidden=hidden, inner=inner)
    if kind == "head":
        hidden, vocab = rng.choice([(4096, 128256), (1536, 32000), (3584, 152064), (256, 32000), (4096, 32064)])
        return dict(kind=kind, rows=_spread(rng, 48, 4096), hidden=hidden, vocab=vocab,
                    weighted=round(rng.uniform(0.3, 1.0), 3))
    if kind == "optimizer":
        return dict(kind=kind, count=8 * _spread(rng, 1 << 13, 27000000), accumulate=rng.random() < 0.5)
    if rng.random() < 0.5:
        return dict(kind=kind, model="tiny", layers=rng.randint(1, 6), rows=rng.randint(1, 6),
                    seq=128 * rng.randint(3, 16), docs="packed")
    return dict(kind=kind, model="qwen2.5-1.5b-image", layers=1, rows=1, seq=128 * rng.randint(16, 36), docs="images")


# ---------------------------------------------------------------------------------------- inputs
def _randn(gen, *shape, scale=1.0):
    return (torch.randn(*shape, generator=gen, device="cuda") * scale).to(BF16)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _rows(case, seed, vocab=1000):
    """Token rows of the named corpus: NumPy arrays, [rows, seq] each."""
    rows, seq, docs = case["rows"], case["seq"], case["docs"]
    if docs == "packed":
        return synthetic.pretraining_rows(rows, seq, vocab, eos_token_id=2, pad_token_id=0, seed=seed)
    if docs == "images":
        text, codes = (151000, 16384) if vocab > 160000 else (600, 300)
        return synthetic.maskgit_rows(rows, seq, text_vocab=text, code_base=vocab - codes - 64, num_codes=codes,
                                      mask_id=vocab - 64, im_start=text + 1, im_end=text + 2, newline_id=198,
                                      pad_token_id=0, seed=seed)
    count = 1 if docs == "one" else 4
    low = seq if count == 1 else seq // 8
    return synthetic.long_document_rows(rows, seq, vocab, docs_per_row=count, min_len=low,
                                        max_len=max(low, seq if count == 1 else 3 * seq // 8), seed=seed)


def _full_rows(case, seed):
    """The same with the padding after a row's last document turned into one more document: every
    position has an output that means something."""
    arrays = _rows(case, seed)
    seg = arrays["segment_ids"]
    arrays["segment_ids"] = np.where(seg == 0, seg.max(axis=1, keepdims=True) + 1, seg)
    return arrays


def _on_gpu(arrays, name):
    return torch.from_numpy(arrays[name]).cuda() if name in arrays else None


def _prepare_attention(case, seed):
    gen, arrays = _generator(seed), _full_rows(case, seed)
    b, s, hq, hkv, d = case["rows"], case["seq"], case["heads"], case["kv_heads"], case["dim"]

    def heads(packed):
        x = packed.view(b, s, hq + 2 * hkv, d)
        return x[:, :, :hq], x[:, :, hq:hq + hkv], x[:, :, hq + hkv:]

    seg, end = _on_gpu(arrays, "segment_ids"), _on_gpu(arrays, "attention_end")
    qkv = _randn(gen, b * s, (hq + 2 * hkv) * d)
    return dict(q=heads(qkv), dout=_randn(gen, b, s, hq, d), dqkv=heads(torch.empty_like(qkv)),
                meta=attention.attention_metadata(torch.ones_like(seg), seg, end)[2])


def _prepare_mlp(case, seed):
    gen = _generator(seed)
    t, d, f = case["tokens"], case["hidden"], case["inner"]
    return dict(x=_randn(gen, t, d), branch=_randn(gen, t, d), dout=_randn(gen, t, d, scale=1e-2),
                norm=1 + _randn(gen, d, scale=0.1), gate_up=_randn(gen, 2 * f, d, scale=0.02),
                down=_randn(gen, d, f, scale=0.02), grads=[torch.zeros(2 * f, d, dtype=BF16, device="cuda"),
                                                         torch.zeros(d, f, dtype=BF16, device="cuda")])


def _prepare_head(case, seed):
    gen = _generator(seed)
    rows, d, vocab = case["rows"], case["hidden"], case["vocab"]
    weights = (torch.rand(rows, generator=gen, device="cuda") < case["weighted"]).float()
    weights[0] = 1.0
    return dict(hidden=_randn(gen, rows, d), head=_randn(gen, vocab, d, scale=0.02), weights=weights,
                targets=torch.randint(0, vocab, (rows,), generator=gen, device="cuda"), scale=1.0 / weights.sum())


def _prepare_optimizer(case, seed):
    gen, n = _generator(seed), case["count"]

    def values(scale):
        out = torch.empty(n, dtype=BF16, device="cuda")
        for at in range(0, n, 1 << 24):
            out[at:at + (1 << 24)] = _randn(gen, min(1 << 24, n - at), scale=scale)
        return out

    p, g, m, v = values(0.02), values(1e-3), values(1e-4), values(1e-3).square_()
    # two vectors without decay (the norms of a layer), then matrices
    cuts = sorted({0, n // 4096 // 8 * 8, n // 2048 // 8 * 8, n // 3 // 8 * 8, n})
    modes = [0 if hi <= n // 2048 else 1 for hi in cuts[1:]]
    return dict(p=p, g=g.float() if case["accumulate"] else g, m=m, v=v,
                bounds=torch.tensor(cuts, dtype=torch.int64, device="cuda"),
                modes=torch.tensor(modes, dtype=torch.int32, device="cuda"))


ADAM = dict(lr=1e-3, b1=0.9, b2=0.95, eps=1e-8, decay=0.1, step=7)


def _prepare_step(case, seed):
    cfg = preset(case["model"], num_hidden_layers=case["layers"])
    params, gen = ModelParams(cfg, BF16, "cuda"), _generator(seed)
    for name, t in params.named_tensors():
        if name.endswith("norm.weight"):
            t.fill_(1.0)
        else:
            t.copy_(_randn(gen, *t.shape, scale=cfg.initializer_range))
    arrays = _rows(case, seed, cfg.vocab_size)
    if cfg.pad_token_id:
        arrays["input_ids"][arrays["attention_mask"] == 0] = cfg.pad_token_id
    batch = {k: torch.from_numpy(v).cuda() for k, v in arrays.items()}
    return dict(cfg=cfg, params=params, batch=batch, engine=LayerwiseEngine(cfg, LocalProvider(params, BF16)))


def prepare(case, seed):
    if case["kind"] == "moba":
        return dict(_prepare_attention(case, seed), case=case)
    made = {"attention": _prepare_attention, "mlp": _prepare_mlp, "head": _prepare_head, "optimizer": _prepare_optimizer,
            "step": _prepare_step}[case["kind"]](case, seed)
    return dict(made, case=case)


# ---------------------------------------------------------------------------------------- one pass
def _run_attention(st):
    q, k, v = st["q"]
    dq, dk, dv = st["dqkv"]
    if st["case"]["kind"] == "moba":
        groups = moba.build_groups(q, k, st["meta"], st["case"]["block"], st["case"]["top_k"])
        out, lse = moba.moba_grouped_forward(q, k, v, st["meta"], groups)
        moba.moba_grouped_backward(q, k, v, out, st["dout"], lse, st["meta"], groups, dq=dq, dk=dk, dv=dv)
    else:
        out, lse = attention.flash_attention_forward(q, k, v, st["meta"])
        attention.flash_attention_backward(q, k, v, out, st["dout"], lse, st["meta"], dq=dq, dk=dk, dv=dv)
    return dict(out=out, lse=lse, dq=dq, dk=dk, dv=dv)


def _run_mlp(st):
    normed, rstd, h = elementwise.rmsnorm_forward(st["x"], st["norm"], 1e-5, residual=st["branch"])
    gate_up = gemm.linear_forward(normed, st["gate_up"])
    act = elementwise.swiglu_forward(gate_up)
    out = gemm.linear_forward(act, st["down"])
    dact = gemm.linear_dgrad(st["dout"], st["down"])
    gemm.linear_wgrad(st["dout"], act, out=st["grads"][1])
    dgate_up = elementwise.swiglu_backward(gate_up, dact)
    dnormed = gemm.linear_dgrad(dgate_up, st["gate_up"])
    gemm.linear_wgrad(dgate_up, normed, out=st["grads"][0])
    dx, dnorm = elementwise.rmsnorm_backward(dnormed, h, st["norm"], rstd, dres=st["dout"])
    return dict(h=h, out=out, dx=dx, dnorm=dnorm, dgate_up=st["grads"][0], ddown=st["grads"][1])


def _run_head(st):
    nll, total, lse, coef = cross_entropy.cut_ce_forward(st["hidden"], st["head"], st["targets"], st["weights"], st["scale"])
    dhidden, dhead = cross_entropy.cut_ce_backward(st["hidden"], st["head"], st["targets"], lse, coef)
    return dict(nll=nll, total=total, lse=lse, dhidden=dhidden, dhead=dhead)


def _run_optimizer(st):
    rounded = st["g"].dtype == F32
    norm = torch.sqrt(elementwise.sum_of_squares(st["g"], round_bf16=rounded))
    clip = torch.clamp(1.0 / norm, max=1.0).reshape(1)
    elementwise.adamw_regions(st["p"], st["g"], st["m"], st["v"], st["bounds"], st["modes"], clip=clip, round_bf16=rounded,
                              **ADAM)
    return dict(norm=norm, p=st["p"], m=st["m"], v=st["v"])


def _run_step(st):
    weights = st["batch"].get("prediction_weights")
    count = st["batch"]["attention_mask"].sum() if weights is None else weights.sum()
    nll, total = st["engine"](st["batch"], 1.0 / count.float(), first=True)
    return dict(nll=nll, total=total, **{name: unit.grad for name, unit in st["params"].units.items()})


def run(state):
    return {"attention": _run_attention, "moba": _run_attention, "mlp": _run_mlp, "head": _run_head,
            "optimizer": _run_optimizer, "step": _run_step}[state["case"]["kind"]](state)


# ---------------------------------------------------------------------------------------- what it cannot do without
def _pairs(arrays):
    """Visible (query, key) pairs of the rows."""
    seg = arrays["segment_ids"]
    idx = np.broadcast_to(np.arange(seg.shape[1]), seg.shape)
    first = np.ones(seg.shape, dtype=bool)
    first[:, 1:] = seg[:, 1:] != seg[:, :-1]
    start = np.maximum.accumulate(np.where(first, idx, 0), axis=1)
    last = np.maximum(idx, arrays["attention_end"]) if "attention_end" in arrays else idx
    return float(np.where(seg != 0, last - start + 1, 0).sum())


def work(case):
    kind = case["kind"]
    if kind in ("attention", "moba"):
        t, hq, hkv, d = case["rows"] * case["seq"], case["heads"], case["kv_heads"], case["dim"]
        arrays = _full_rows(case, 0)
        if kind == "attention":
            pairs = _pairs(arrays)
        else:
            pairs = 0.0
            for n in np.unique(arrays["segment_ids"], return_counts=True)[1].tolist():
                at = np.arange(n)
                pairs += float((at % case["block"] + 1 + np.minimum(at // case["block"], case["top_k"] - 1) * case["block"]).sum())
        # q, dout, out, dq and k, v, dk, dv once each, and the log-sum-exp
        return dict(bytes=8.0 * t * (hq + hkv) * d + 4.0 * t * hq, flops=14.0 * pairs * hq * d)
    if kind == "mlp":
        t, d, f = case["tokens"], case["hidden"], case["inner"]
        return dict(bytes=2.0 * (6 * t * d + 6 * d * f), flops=18.0 * t * d * f)
    if kind == "head":
        rows, d, vocab = case["rows"], case["hidden"], case["vocab"]
        return dict(bytes=2.0 * (2 * rows * d + 2 * vocab * d), flops=6.0 * rows * d * vocab)
    if kind == "optimizer":
        return dict(bytes=(12.0 + (4 if case["accumulate"] else 2)) * case["count"], flops=16.0 * case["count"])
    cfg = preset(case["model"], num_hidden_layers=case["layers"])
    t, d, q, kv = case["rows"] * case["seq"], cfg.hidden_size, cfg.query_width, cfg.key_value_width
    layer = d * q + 2 * d * kv + q * d + 3 * d * cfg.intermediate_size
    rows = t
    if case["docs"] == "images":
        rows = float((_rows(case, 0, cfg.vocab_size)["prediction_weights"] > 0).sum())
    flops = 6.0 * (t * case["layers"] * layer + rows * cfg.vocab_size * d)
    flops += 14.0 * case["layers"] * q * _pairs(_rows(case, 0, cfg.vocab_size))
    # weights read and gradients written once
    return dict(bytes=4.0 * (case["layers"] * layer + 2 * cfg.vocab_size * d), flops=flops)


def tolerance(case):
    # bf16 results of fp32 accumulation: about four times what two correct orders of summation differ by
    # (measured against 64 bits: attention 0.0025, moba 0.003, mlp 0.0058, head 0.0027, optimizer 0.0017, step 0.01)
    return {"attention": dict(rel=1e-2, max=0.4), "moba": dict(rel=1e-2, max=0.6), "mlp": dict(rel=1.5e-2, max=0.6),
            "head": dict(rel=1e-2, max=0.4), "optimizer": dict(rel=5e-3, max=0.1), "step": dict(rel=2.5e-2, max=0.95)}[case["kind"]]


# ---------------------------------------------------------------------------------------- the same in 64 bits
def _exact_attention_head(q, k, v, dout, see, scale):
    """One head with its visibility mask ``see`` ([n, m] bool): out, lse, dq, dk, dv."""
    s = (q @ k.T).mul_(scale).masked_fill_(~see, -math.inf)
    lse = torch.logsumexp(s, dim=1)
    empty = torch.isinf(lse)
    lse = torch.where(empty, torch.zeros_like(lse), lse)
    p = s.sub_(lse[:, None]).exp_()
    out = p @ v
    dv = p.T @ dout
    ds = (dout @ v.T).sub_((out * dout).sum(1, keepdim=True)).mul_(p).mul_(scale)
    return out, lse, ds @ k, ds.T @ q, dv


def _exact_attention(case, st, arrays):
    q, k, v = (x.to(F64) for x in st["q"])
    dout = st["dout"].to(F64)
    b, s, hq, _ = q.shape
    group = hq // k.shape[2]
    out, dq, dk, dv = torch.zeros_like(q), torch.zeros_like(q), torch.zeros_like(k), torch.zeros_like(v)
    lse = torch.zeros(b, hq, s, dtype=F64, device="cuda")
    scale = 1.0 / math.sqrt(case["dim"])
    seg = torch.from_numpy(arrays["segment_ids"]).cuda()
    end = _on_gpu(arrays, "attention_end")
    for bi in range(b):
        bounds = [0] + (torch.nonzero(seg[bi, 1:] != seg[bi, :-1]).reshape(-1) + 1).tolist() + [s]
        for lo, hi in zip(bounds[:-1], bounds[1:]):
            if int(seg[bi, lo]) == 0:
                continue
            at = torch.arange(hi - lo, device="cuda")
            last = at if end is None else torch.maximum(at, end[bi, lo:hi].long() - lo)
            see = at[None, :] <= last[:, None]
            rows = slice(lo, hi)
            for h in range(hq):
                j = h // group
                mine = see
                if case["kind"] == "moba":
                    block, n = case["block"], hi - lo
                    own = at // block
                    whole = n // block
                    chosen = torch.zeros(n, n // block + 1, dtype=torch.bool, device="cuda")
                    chosen.scatter_(1, own[:, None], True)
                    if whole:
                        means = k[bi, lo:lo + whole * block, j].reshape(whole, block, -1).mean(1)
                        gate = (q[bi, rows, h] @ means.T).masked_fill_(torch.arange(whole, device="cuda")[None] >= own[:, None], -math.inf)
                        best = gate.topk(min(case["top_k"] - 1, whole), dim=1)
                        chosen.scatter_(1, best.indices, chosen.gather(1, best.indices) | ~torch.isinf(best.values))
                    mine = see & chosen[:, own]
                o, l, a, c, e = _exact_attention_head(q[bi, rows, h], k[bi, rows, j], v[bi, rows, j], dout[bi, rows, h], mine, scale)
                out[bi, rows, h], lse[bi, h, rows], dq[bi, rows, h] = o, l, a
                dk[bi, rows, j] += c
                dv[bi, rows, j] += e
    return dict(out=out, lse=lse, dq=dq, dk=dk, dv=dv)


def _exact_mlp(case, st):
    w = {n: st[n].to(F64).requires_grad_() for n in ("norm", "gate_up", "down")}
    h = (st["x"].to(F64) + st["branch"].to(F64)).requires_grad_()
    normed = h * torch.rsqrt(h.square().mean(1, keepdim=True) + 1e-5) * w["norm"]
    gate, up = (normed @ w["gate_up"].T).chunk(2, dim=1)
    out = (torch.nn.functional.silu(gate) * up) @ w["down"].T
    dh, dnorm, dgate_up, ddown = torch.autograd.grad(out, [h, w["norm"], w["gate_up"], w["down"]], st["dout"].to(F64))
    return dict(h=h.detach(), out=out.detach(), dx=dh + st["dout"].to(F64), dnorm=dnorm, dgate_up=dgate_up, ddown=ddown)


def _exact_head(case, st):
    hidden, head = st["hidden"].to(F64), st["head"].to(F64)
    logits = hidden @ head.T
    lse = torch.logsumexp(logits, dim=1)
    weights, targets = st["weights"].to(F64), st["targets"][:, None]
    nll = ((lse - logits.gather(1, targets)[:, 0]) * weights).sum()
    g = logits.sub_(lse[:, None]).exp_()
    g.scatter_add_(1, targets, torch.full_like(targets, -1, dtype=F64))
    g *= (weights * st["scale"].to(F64))[:, None]
    return dict(nll=nll, total=weights.sum(), lse=lse, dhidden=g @ head, dhead=g.T @ hidden)


def _exact_optimizer(case, st):
    p, g, m, v = (st[n].to(BF16).to(F64) for n in "pgmv")
    norm = g.square().sum().sqrt()
    g *= torch.clamp(1.0 / norm, max=1.0)
    m = m * ADAM["b1"] + (1 - ADAM["b1"]) * g
    v = v * ADAM["b2"] + (1 - ADAM["b2"]) * g * g
    new = (m / (1 - ADAM["b1"] ** ADAM["step"])) / ((v / (1 - ADAM["b2"] ** ADAM["step"])).sqrt() + ADAM["eps"])
    for lo, hi, mode in zip(st["bounds"].tolist()[:-1], st["bounds"].tolist()[1:], st["modes"].tolist()):
        new[lo:hi] += ADAM["decay"] * mode * p[lo:hi]
    return dict(norm=norm, p=p - ADAM["lr"] * new, m=m, v=v)


def _exact_step(case, st):
    cfg, batch = st["cfg"], st["batch"]
    flat = {n: u.data.to(F64).requires_grad_() for n, u in st["params"].units.items()}
    view = {n: {s.name: flat[n][s.offset:s.offset + s.numel].view(s.shape) for s in u.layout.segments}
            for n, u in st["params"].units.items()}
    ids, seg = batch["input_ids"].long(), batch["segment_ids"].long()
    b, s = ids.shape
    hq, hkv, d = cfg.num_attention_heads, cfg.num_key_value_heads, cfg.head_dim
    at = torch.arange(s, device="cuda")
    end = batch.get("attention_end")
    last = at.expand(b, s) if end is None else torch.maximum(at.expand(b, s), end.long())
    see = (seg[:, :, None] == seg[:, None, :]) & (seg[:, :, None] != 0) & (at[None, None, :] <= last[:, :, None])
    freq = cfg.rope_theta ** (-torch.arange(0, d, 2, dtype=F64, device="cuda") / d)
    angle = batch["position_ids"].to(F64)[:, :, None] * freq
    cos, sin = (f(angle).to(BF16).to(F64)[:, :, None, :] for f in (torch.cos, torch.sin))   # the table is bf16 by definition

    def norm(x, w):
        return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + cfg.rms_norm_eps) * w

    def rotate(x):
        x1, x2 = x[..., :d // 2], x[..., d // 2:]
        return torch.cat((x1 * cos - x2 * sin, x2 * cos + x1 * sin), dim=-1)

    table = view["embed"]["embed"]
    h = torch.nn.functional.embedding(ids, table)
    keep = (ids != cfg.pad_token_id)[:, :, None]
    h = torch.where(keep, h, h.detach())
    for i in range(cfg.num_hidden_layers):
        w = view["layer.%d" % i]
        qkv = norm(h, w["ln1"]) @ w["qkv_w"].T
        if "qkv_b" in w:
            qkv = qkv + w["qkv_b"]
        qkv = qkv.view(b, s, hq + 2 * hkv, d)
        q, k, v = rotate(qkv[:, :, :hq]), rotate(qkv[:, :, hq:hq + hkv]), qkv[:, :, hq + hkv:]
        heads = []
        for j in range(hq):
            score = torch.einsum("bqd,bkd->bqk", q[:, :, j], k[:, :, j * hkv // hq]) / math.sqrt(d)
            p = torch.softmax(score.masked_fill(~see, -1e300), dim=-1) * see
            heads.append(p @ v[:, :, j * hkv // hq])
        h = h + torch.stack(heads, dim=2).reshape(b, s, hq * d) @ w["o_w"].T
        gate, up = (norm(h, w["ln2"]) @ w["gu_w"].T).chunk(2, dim=-1)
        h = h + (torch.nn.functional.silu(gate) * up) @ w["down_w"].T
    y = norm(h, view["final"]["norm"])
    if "prediction_weights" in batch:
        weights, targets = batch["prediction_weights"].to(F64), batch["prediction_targets"].long()
        count = weights.sum()
    else:
        weights = torch.zeros(b, s, dtype=F64, device="cuda")
        weights[:, :-1] = ((seg[:, 1:] == seg[:, :-1]) & (seg[:, 1:] != 0)).to(F64)
        targets = torch.cat((ids[:, 1:], ids[:, :1]), dim=1)
        count = batch["attention_mask"].sum()
    pick = weights.reshape(-1) > 0
    logits = y.reshape(b * s, -1)[pick] @ view["final"]["lm_head"].T
    chosen = logits.gather(1, targets.reshape(-1)[pick][:, None])[:, 0]
    nll = ((torch.logsumexp(logits, dim=1) - chosen) * weights.reshape(-1)[pick]).sum()
    names = list(flat)
    grads = torch.autograd.grad(nll / count, [flat[n] for n in names])
    return dict(nll=nll.detach(), total=weights.sum(), **dict(zip(names, grads)))


def exact(case, seed):
    st = prepare(case, seed)
    if case["kind"] in ("attention", "moba"):
        return _exact_attention(case, st, _full_rows(case, seed))
    return {"mlp": _exact_mlp, "head": _exact_head, "optimizer": _exact_optimizer, "step": _exact_step}[case["kind"]](case, st)
