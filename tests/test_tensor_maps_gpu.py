"""Launches whose tensor maps leave the cache while the launch still collects the others: the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limit", [1, 2, 3])
def test_a_full_cache_is_emptied_between_two_lookups_of_a_launch(cuda_lib, limit):
    from causal_trainer_dev_b200.ops import attention as A
    from causal_trainer_dev_b200.ops import gemm as G

    gen = torch.Generator(device="cuda").manual_seed(1)
    bf16 = lambda *s: torch.randn(*s, generator=gen, device="cuda").bfloat16()  # noqa: E731
    products = [(bf16(m, k), bf16(n, k)) for m, n, k in ((64, 1536, 8960), (333, 4096, 512), (1024, 1536, 17920), (4096, 4096, 4096))]
    q, k, v, do = bf16(2, 256, 4, 64), bf16(2, 256, 2, 64), bf16(2, 256, 2, 64), bf16(2, 256, 4, 64)
    meta = A.build_attention_meta(torch.ones(2, 256, dtype=torch.int32, device="cuda"))

    def run():
        o, lse = A.flash_attention_forward(q, k, v, meta)
        out = [o, lse, *A.flash_attention_backward(q, k, v, o, do, lse, meta)]
        for a, b in products:
            out += [G.gemm(a, b), G.gemm(a, b, out_dtype=torch.float32)]
        return out

    want = run()
    before = cuda_lib.lib().ctb_tensor_map_limit(limit)
    try:
        for _ in range(2):
            assert all(torch.equal(a, b) for a, b in zip(run(), want))
    finally:
        assert cuda_lib.lib().ctb_tensor_map_limit(before) == limit
    for (a, b), got in zip(products, want[6::2]):
        ref = a.double() @ b.double().t()
        assert ((got.double() - ref).norm() / ref.norm()).item() < 1e-5
    assert cuda_lib.device_status() == (0, 0, 0, 0)
