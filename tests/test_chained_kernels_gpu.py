"""Chained launches (csrc/host_common.h) behind a long predecessor that lets its successors start at once: on a side stream, over
two streams and under capture they give the bits of the same calls with the host waiting between any two."""
import pytest
import torch

pytestmark = pytest.mark.gpu

TOKENS, WIDE, F, D, HEADS, KV, DIM, VOCAB = 512, 16384, 8960, 1536, 8, 2, 64, 1000
QKV = (HEADS + 2 * KV) * DIM


def _randn(gen, *shape, scale=1.0):
    return (torch.randn(*shape, generator=gen, device="cuda") * scale).bfloat16()


def _inputs():
    from causal_trainer_dev_b200.ops import attention as A
    from causal_trainer_dev_b200.ops import elementwise as E

    gen = torch.Generator(device="cuda").manual_seed(7)
    pos = torch.arange(TOKENS, device="cuda").repeat(1, 1)
    cos, sin = E.rope_table(pos, E.inverse_frequencies(DIM, 1e4, device="cuda"))
    return dict(
        gate_up=_randn(gen, WIDE, 2 * F), norm=_randn(gen, F), norm2=_randn(gen, D), w_in=_randn(gen, D, F, scale=0.02),
        w_gu=_randn(gen, 2 * D, D, scale=0.02), w_qkv=_randn(gen, QKV, D, scale=0.02), bias=_randn(gen, QKV),
        head=_randn(gen, VOCAB, D, scale=0.05), cos=cos, sin=sin, meta=A.build_attention_meta((pos // 200 + 1).int()),
        ids=torch.randint(0, VOCAB, (1, TOKENS), generator=gen, device="cuda"), weights=torch.rand(TOKENS, device="cuda"),
        scale=torch.tensor(0.37, device="cuda"), dout=_randn(gen, 1, TOKENS, HEADS, DIM), table=torch.empty(VOCAB, D, device="cuda"))


def _steps(x, wide, out):
    """The calls, as a generator: each step reads what the one before it has just written.  ``wide`` receives the long
    predecessor's result, of which the last rows are read first; ``out`` collects what is compared."""
    from causal_trainer_dev_b200.ops import attention as A
    from causal_trainer_dev_b200.ops import cross_entropy as CE
    from causal_trainer_dev_b200.ops import elementwise as E
    from causal_trainer_dev_b200.ops import lib as L
    from causal_trainer_dev_b200.ops.gemm import gemm

    def long_one():
        code = L.lib().ctb_swiglu_fwd(x["gate_up"].data_ptr(), wide.data_ptr(), WIDE, F, L.raw_stream())
        L.check(code, "ctb_swiglu_fwd")

    tail = wide[WIDE - TOKENS:]
    long_one()
    yield
    normed, rstd, _ = E.rmsnorm_forward(tail, x["norm"], 1e-5)
    yield
    hidden = gemm(normed, x["w_in"])                                   # long K: parts of it on several CTAs
    yield
    gu = gemm(hidden, x["w_gu"])
    yield
    act = E.swiglu_forward(gu)
    yield
    dgu = E.swiglu_backward(gu, act)
    yield
    h2, rstd2, summed = E.rmsnorm_forward(act, x["norm2"], 1e-5, residual=hidden)
    yield
    qkv = gemm(h2, x["w_qkv"], bias=x["bias"])
    yield
    E.rope_inplace(qkv, x["cos"], x["sin"], HEADS + KV, DIM, DIM, "gpt-neox")
    yield
    packed = qkv.view(1, TOKENS, HEADS + 2 * KV, DIM)
    q, k, v = packed[:, :, :HEADS], packed[:, :, HEADS:HEADS + KV], packed[:, :, HEADS + KV:]
    o, lse = A.flash_attention_forward(q, k, v, x["meta"])
    yield
    dqkv = torch.empty_like(packed)
    A.flash_attention_backward(q, k, v, o, x["dout"], lse, x["meta"], dq=dqkv[:, :, :HEADS], dk=dqkv[:, :, HEADS:HEADS + KV],
                               dv=dqkv[:, :, HEADS + KV:])
    yield
    dbias = torch.empty(QKV, device="cuda")
    E.column_sum(dqkv.view(TOKENS, QKV), dbias)
    yield
    dh = gemm(dqkv.view(TOKENS, QKV), x["w_qkv"], b_mn=True)
    yield
    dx, dw = E.rmsnorm_backward(dh, summed, x["norm2"], rstd2, dres=act)
    yield
    nll, total, dhid, dhead = CE.cut_ce_forward_backward(dx, x["head"], x["ids"][0], x["weights"], x["scale"])
    yield
    nll2, _, lse2, coef = CE.cut_ce_forward(dhid, x["head"], x["ids"][0], x["weights"], x["scale"])
    yield
    x["table"].zero_()
    E.embedding_backward(x["ids"], dhid, x["table"], pad_id=5)
    yield
    long_one()                                                         # once more: the norm must not see the first one's rows
    yield
    again = E.rmsnorm_backward(tail, tail, x["norm"], rstd)
    out += [normed, hidden, act, dgu, h2, qkv, o, lse, dqkv, dbias, dh, dx, dw, nll, total, dhid, dhead, nll2, lse2, coef,
            x["table"], *again]


def _spoil(wide):
    wide.fill_(3.0)
    torch.cuda.synchronize()


def test_the_bits_of_a_sequence_that_the_host_waits_in(cuda_lib):
    x = _inputs()
    assert cuda_lib.lib().ctb_attn_bwd_workspace(1, TOKENS, TOKENS, HEADS, KV, DIM) > 0      # dK / dV in parts among them
    wide = torch.empty(WIDE, F, dtype=torch.bfloat16, device="cuda")
    want = []
    _spoil(wide)
    for _ in _steps(x, wide, want):
        torch.cuda.synchronize()
    torch.cuda.synchronize()
    want = [t.clone() for t in want]
    assert all(bool(torch.isfinite(t.float()).all()) for t in want)

    def same(got, how):
        torch.cuda.synchronize()
        assert cuda_lib.device_status() == (0, 0, 0, 0)
        off = [i for i, (a, b) in enumerate(zip(want, got, strict=True)) if not torch.equal(a, b)]
        assert not off, (how, off)

    side, other = torch.cuda.Stream(), torch.cuda.Stream()
    for turn in range(4):
        got = []
        _spoil(wide)
        with torch.cuda.stream(side):
            for _ in _steps(x, wide, got):
                pass
        same(got, f"one stream, {turn}")
        # every other step on a second stream
        got = []
        _spoil(wide)
        streams, steps = [side, other], _steps(x, wide, got)
        for i in range(1000):
            now, then = streams[i % 2], streams[(i + 1) % 2]
            now.wait_stream(then)
            with torch.cuda.stream(now):
                if next(steps, "done") == "done":
                    break
        side.wait_stream(other)
        same(got, f"two streams, {turn}")

    def captured(streams):
        got, graph = [], torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            main = torch.cuda.current_stream()
            steps, use = _steps(x, wide, got), [main, *streams]
            for i in range(1000):
                now, then = use[i % len(use)], use[(i - 1) % len(use)]
                if i and now is not then:
                    now.wait_stream(then)
                with torch.cuda.stream(now):
                    if next(steps, "done") == "done":
                        break
            for s in streams:
                main.wait_stream(s)
        for turn in range(3):
            for t in got:
                t.zero_()
            _spoil(wide)
            graph.replay()
            same(got, f"captured over {len(use)} streams, {turn}")

    captured([])
    captured([other])


def test_a_refused_launch_leaves_no_error_behind(cuda_lib):
    """An empty grid is refused; whoever launches next, the framework's own kernels among them, must not be told of it."""
    from causal_trainer_dev_b200.ops import elementwise as E

    x, w = torch.empty(0, 256, device="cuda", dtype=torch.bfloat16), torch.ones(256, device="cuda", dtype=torch.bfloat16)
    for _ in range(2):
        with pytest.raises(cuda_lib.KernelError):
            E.rmsnorm_forward(x, w, 1e-5)
        assert float(torch.ones(300, device="cuda").cumsum(0)[-1]) == 300


@pytest.mark.parametrize("captured", [False, True])
def test_an_event_between_two_launches_is_waited_for(cuda_lib, captured):
    """The kernel before a chained one lets its successor start at once; what the chained one reads comes from another stream,
    whose event its own stream waits for in between, and is still being written."""
    from causal_trainer_dev_b200.ops import elementwise as E
    from causal_trainer_dev_b200.ops import lib as L
    from causal_trainer_dev_b200.ops.gemm import gemm

    gen = torch.Generator(device="cuda").manual_seed(8)
    gate_up, w = _randn(gen, WIDE, 2 * F), _randn(gen, F)
    weight, short = _randn(gen, 256, F, scale=0.02), _randn(gen, 512, 2 * F)
    wide, act = torch.empty(WIDE, F, dtype=torch.bfloat16, device="cuda"), torch.empty(512, F, dtype=torch.bfloat16, device="cuda")
    tail = wide[WIDE - 512:]
    main, other = torch.cuda.Stream(), torch.cuda.Stream()

    def into(gu, out, rows):
        L.check(L.lib().ctb_swiglu_fwd(gu.data_ptr(), out.data_ptr(), rows, F, L.raw_stream()), "ctb_swiglu_fwd")

    def calls(s):
        other.wait_stream(s)
        with torch.cuda.stream(other):
            into(gate_up, wide, WIDE)                                  # about 80 us
        into(short, act, 512)                                          # lets its successor in, and is over long before
        s.wait_stream(other)
        normed, rstd, _ = E.rmsnorm_forward(tail, w, 1e-5)
        # the same in front of a product (operands by bulk copies)
        other.wait_stream(s)
        with torch.cuda.stream(other):
            torch.mul(wide, 2.0, out=wide)
        into(short, act, 512)
        s.wait_stream(other)
        return normed, rstd, gemm(tail, weight)

    wide.fill_(3.0)
    into(gate_up, wide, WIDE)
    torch.cuda.synchronize()
    want = list(E.rmsnorm_forward(tail, w, 1e-5)[:2])
    wide.mul_(2.0)
    want.append(gemm(tail, weight))
    torch.cuda.synchronize()
    if captured:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=main):
            got = calls(main)
    for _ in range(5):
        wide.fill_(3.0)
        torch.cuda.synchronize()
        if captured:
            graph.replay()
        else:
            with torch.cuda.stream(main):
                got = calls(main)
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    assert cuda_lib.device_status() == (0, 0, 0, 0)
