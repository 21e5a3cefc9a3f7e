"""Attention kernels whose bounded waits run out while their CTAs go from work item to work item: every warp leaves, the status
says where, and the next launch is right."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(b, s, hq, hkv, d):
    gen = torch.Generator(device="cuda").manual_seed(s)
    # keys and values are the halves of one gathered buffer
    kv = torch.randn(b, s, 2 * hkv * d, generator=gen, device="cuda").bfloat16()
    k, v = (x.unflatten(2, (hkv, d)) for x in kv.split(hkv * d, dim=2))
    q, do = (torch.randn(b, s, hq, d, generator=gen, device="cuda").bfloat16() for _ in range(2))
    return q, k, v, do


@pytest.mark.parametrize("landed", [0, 3, 9])
def test_keys_that_never_land(cuda_lib, landed):
    """Items that see only the first key tiles finish, the others wait for a flag that nothing sets (a limit of about 1 ms)."""
    from causal_trainer_dev_b200.ops import attention as A

    b, s, hq, hkv, d = 1, 2048, 32, 8, 128                       # 256 work items
    q, k, v, _ = _inputs(b, s, hq, hkv, d)
    meta = A.build_attention_meta(torch.ones(b, s, dtype=torch.int32, device="cuda"))
    row = 2 * hkv * d
    flags = torch.zeros(s // 128, dtype=torch.int32, device="cuda")
    flags[:landed] = 1
    A.flash_attention_forward(q, k, v, meta, spin_budget=2_000_000, kv_flags=(flags, 128 * row, row, 1))
    code, *_ = cuda_lib.device_status(raise_on_error=False)
    # the producer gives up, or one of the roles behind it at the same moment
    assert code in (0x0203, 0x0204, 0x0205, 0x0206, 0x0207, 0x0208)
    want = A.flash_attention_forward(q, k, v, meta)
    flags.fill_(1)
    got = A.flash_attention_forward(q, k, v, meta, kv_flags=(flags, 128 * row, row, 1))
    assert all(torch.equal(x, y) for x, y in zip(got, want))
    assert cuda_lib.device_status() == (0, 0, 0, 0)


@pytest.mark.parametrize("d,hq,hkv", [(128, 8, 2), (64, 12, 2)])
def test_every_role_may_give_up_first(cuda_lib, d, hq, hkv):
    """With next to no limit any wait of any warp may be the first that runs out."""
    from causal_trainer_dev_b200.ops import attention as A

    q, k, v, do = _inputs(6, 1152, hq, hkv, d)
    meta = A.build_attention_meta(torch.ones(6, 1152, dtype=torch.int32, device="cuda"))
    o, lse = A.flash_attention_forward(q, k, v, meta)
    want = (o, lse, *A.flash_attention_backward(q, k, v, o, do, lse, meta))
    for _ in range(10):
        A.flash_attention_forward(q, k, v, meta, spin_budget=1)
        fwd = cuda_lib.device_status(raise_on_error=False)[0]
        A.flash_attention_backward(q, k, v, o, do, lse, meta, spin_budget=1)
        bwd = cuda_lib.device_status(raise_on_error=False)[0]
        assert fwd == 0 or 0x0201 <= fwd <= 0x0208
        assert bwd == 0 or 0x0301 <= bwd <= 0x0309
    o2, lse2 = A.flash_attention_forward(q, k, v, meta)
    got = (o2, lse2, *A.flash_attention_backward(q, k, v, o, do, lse, meta))
    assert all(torch.equal(x, y) for x, y in zip(got, want))
    assert cuda_lib.device_status() == (0, 0, 0, 0)
