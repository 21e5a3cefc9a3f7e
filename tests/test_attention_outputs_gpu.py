"""Attention backward with outputs and arguments in the forms that callers may hand in: the same bits as the plain call."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(b, s, hq, hkv, d):
    from causal_trainer_dev_b200.ops import attention as A

    gen = torch.Generator(device="cuda").manual_seed(s)
    q, k, v, do = (torch.randn(b, s, h, d, generator=gen, device="cuda").bfloat16() for h in (hq, hkv, hkv, hq))
    seg = torch.ones(b, s, dtype=torch.int32, device="cuda")
    seg[:, s // 3:] = 2
    meta = A.build_attention_meta(seg)
    o, lse = A.flash_attention_forward(q, k, v, meta)
    return A, q, k, v, do, meta, o, lse


@pytest.mark.parametrize("place", ["q", "dout", "out", "beside q"])
@pytest.mark.parametrize("b,s,hq,hkv,d", [(1, 128, 2, 2, 64), (4, 1152, 12, 2, 128), (3, 2048, 8, 2, 64)])
def test_dq_in_the_place_of_an_input(cuda_lib, place, b, s, hq, hkv, d):
    A, q, k, v, do, meta, o, lse = _case(b, s, hq, hkv, d)
    want = A.flash_attention_backward(q, k, v, o, do, lse, meta)
    for _ in range(3):
        if place == "beside q":                      # halves of one buffer's rows: no byte is shared
            both = torch.cat([q, torch.zeros_like(q)], dim=2).view(b, s, -1)
            qc, dq = (x.unflatten(2, (hq, d)) for x in both.split(hq * d, dim=2))
            doc, oc = do, o
        else:
            qc, doc, oc = q.clone(), do.clone(), o.clone()
            dq = {"q": qc, "dout": doc, "out": oc}[place]
        got = A.flash_attention_backward(qc, k, v, oc, doc, lse, meta, dq=dq)
        assert got[0] is dq and all(torch.equal(x, y) for x, y in zip(got, want))
        if place == "beside q":
            assert torch.equal(qc, q)
    assert cuda_lib.device_status() == (0, 0, 0, 0)


def test_statistics_in_the_place_of_the_log_sum_exp(cuda_lib):
    from causal_trainer_dev_b200.ops.elementwise import attention_backward_stats

    A, q, k, v, do, meta, o, lse = _case(2, 256, 4, 2, 64)
    want = A.flash_attention_backward(q, k, v, o, do, lse, meta)
    got = A.flash_attention_backward(q, k, v, o, do, None, meta, stats=attention_backward_stats(o, do, lse),
                                     spin_budget=np.int64(0))
    assert all(torch.equal(x, y) for x, y in zip(got, want))
    flags = torch.ones(4, dtype=torch.int32, device="cuda")
    kv = torch.cat([k.flatten(2), v.flatten(2)], dim=2)
    kg, vg = (x.unflatten(2, (2, 64)) for x in kv.split(128, dim=2))
    again = A.flash_attention_forward(q, kg, vg, meta, spin_budget=np.int64(0),
                                      kv_flags=(flags, np.int64(128 * 256), np.int64(256), np.int64(1)))
    assert torch.equal(again[0], o) and torch.equal(again[1], lse)
    assert cuda_lib.device_status() == (0, 0, 0, 0)
