"""A product whose kernel wants a workspace that there is no memory for."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_no_memory_for_the_workspace(cuda_lib, monkeypatch, dtype):
    from causal_trainer_dev_b200.ops import gemm as G

    m, n, k = 1000, 1536, 17920
    assert cuda_lib.lib().ctb_gemm_workspace(m, n, k, 0, int(dtype == torch.float32), 0) > 0
    gen = torch.Generator(device="cuda").manual_seed(1)
    a, b = (torch.randn(r, k, generator=gen, device="cuda").bfloat16() for r in (m, n))
    want = a.double() @ b.double().t()
    # one rounding to bf16; or sums that grow by 16 products at a time and are cut to 24 bits each time (towards zero, so the
    # errors of a long K add up: 3e-5 measured in one piece, under 1e-5 in three)
    bound = 2.0 ** -8 if dtype == torch.bfloat16 else k / 16 * 2.0 ** -23
    out = G.gemm(a, b, out_dtype=dtype)
    assert ((out.double() - want).norm() / want.norm()).item() < bound
    empty, refused = torch.empty, []

    def refuse(*args, **kw):
        if kw.get("dtype") == torch.uint8:
            refused.append(args)
            raise torch.cuda.OutOfMemoryError("refused by the test")
        return empty(*args, **kw)

    monkeypatch.setattr(torch, "empty", refuse)
    out = G.gemm(a, b, out_dtype=dtype)
    monkeypatch.undo()
    assert len(refused) == 1 and ((out.double() - want).norm() / want.norm()).item() < bound
    assert cuda_lib.device_status() == (0, 0, 0, 0)
