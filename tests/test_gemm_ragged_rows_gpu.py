"""Products whose last 32-row pieces lie behind the matrix, over several tiles a CTA: a piece without rows stages nothing, so the
stores of the tile before keep their staging blocks.  Every element against 64 bits: a block that is overwritten while it is
read holds another tile's values, which no rounding explains, and a norm over the matrix might not show it.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture
def one_cta(cuda_lib):
    before = cuda_lib.lib().ctb_gemm_set_pair(0)
    yield
    cuda_lib.lib().ctb_gemm_set_pair(before)


def _within(out, a, b):
    """One rounding to the output's type, and fp32 sums of K products whose sizes are those of |a| |b|."""
    want = a.double() @ b.double().t()
    rounding = 2.0 ** -8 if out.dtype == torch.bfloat16 else 2.0 ** -23
    bound = rounding * want.abs() + a.shape[1] * 2.0 ** -24 * (a.double().abs() @ b.double().abs().t())
    return bool(((out.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("k", [8, 72, 520])            # short: the next accumulator is ready at once
@pytest.mark.parametrize("m", [1, 33, 129, 224, 333])  # one to three warps of the last 128 rows have none
def test_warps_without_rows_leave_the_staging_alone(cuda_lib, one_cta, m, k, dtype):
    from causal_trainer_dev_b200.ops import gemm as G

    gen = torch.Generator(device="cuda").manual_seed(m + k)
    n = 32008 if m > 128 else 64008                       # two tiles a CTA and more
    a, b = (torch.randn(r, k, generator=gen, device="cuda").bfloat16() for r in (m, n))
    for _ in range(3):
        out = torch.full((m + 2, n), 7.0, dtype=dtype, device="cuda")
        G.gemm(a, b, out=out[:m])
        assert _within(out[:m], a, b) and bool((out[m:] == 7).all())
    assert cuda_lib.device_status() == (0, 0, 0, 0)


@pytest.mark.parametrize("ids", [torch.int32, torch.int64])
@pytest.mark.parametrize("rows,vocab,d,tm", [
    (333, 32000, 64, None), (33, 64008, 512, None), (200, 40000, 128, None),                     # one CTA
    (1100, 32000, 512, 1), (4000, 5000, 256, 1), (644, 6216, 584, 2), (2077, 2064, 608, 2)])     # two, 256 or 512 rows
def test_kept_logits_and_their_gradients(cuda_lib, rows, vocab, d, tm, ids):
    """The loss epilogues, on the kernel that the sizes choose."""
    import ctypes

    form = (ctypes.c_int * 4)()
    for gradients in (0, 1):
        assert (form[0] if cuda_lib.lib().ctb_ce_pair_choice(rows, vocab, d, gradients, form) else None) == tm
    gen = torch.Generator(device="cuda").manual_seed(rows)
    hidden = torch.randn(rows, d, generator=gen, device="cuda").bfloat16()
    head = (torch.randn(vocab, d, generator=gen, device="cuda") * 0.05).bfloat16()
    targets = torch.randint(0, vocab, (rows,), generator=gen, device="cuda", dtype=ids)
    step = targets.element_size() // 4
    p, ln, slabs = cuda_lib.ptr, ctypes.c_long, -(-vocab // 256)
    none = (None, ln(0), ln(0), ctypes.c_uint(0))
    want = hidden.double() @ head.double().t()
    lse = torch.logsumexp(want, -1)
    size = d * 2.0 ** -24 * (hidden.double().abs() @ head.double().abs().t())       # error of a logit
    for _ in range(3):
        pmax, psum = (torch.empty(slabs, rows, device="cuda") for _ in range(2))
        at_target, logits = torch.zeros(rows, device="cuda"), torch.full((rows + 2, vocab), 7.0, device="cuda")
        assert cuda_lib.lib().ctb_ce_stats(p(hidden), p(head), rows, vocab, d, ln(d), ln(d), p(targets), step, p(pmax),
                                           p(psum), p(at_target), *none, *none, 0, 0, p(logits), ln(vocab), cuda_lib.stream_ptr()) == 0
        assert bool(((logits[:rows].double() - want).abs() <= size + 2.0 ** -23 * want.abs()).all())
        assert bool((logits[rows:] == 7).all())
        assert torch.equal(at_target, logits[:rows].gather(1, targets.long()[:, None])[:, 0])
        g = torch.full((rows + 2, vocab), 7.0, device="cuda", dtype=torch.bfloat16)
        coef = torch.ones(rows, device="cuda")
        assert cuda_lib.lib().ctb_ce_dlogits(p(hidden), p(head), p(g), rows, vocab, d, ln(d), ln(d), ln(vocab), p(targets), step,
                                             p(lse.float()), p(coef), 0, cuda_lib.stream_ptr()) == 0
        prob = (want - lse[:, None]).exp()
        exact = prob.clone()
        exact[torch.arange(rows, device="cuda"), targets.long()] -= 1
        # the exponential's argument is off by the logit's error and by one rounding of the log-sum-exp and of the difference
        wrong = prob * (size + 2.0 ** -23 * (want.abs() + 2 * lse.abs()[:, None]) + 2.0 ** -21)
        assert bool(((g[:rows].double() - exact).abs() <= 2.0 ** -8 * exact.abs() + wrong).all())
        assert bool((g[rows:] == 7).all())
    assert cuda_lib.device_status() == (0, 0, 0, 0)
