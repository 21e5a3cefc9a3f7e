"""The sort of token ids behind the embedding gradient against a stable sort."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 500, 1024, 1025, 2047, 2048])
@pytest.mark.parametrize("values", [1, 7, 1 << 31])
def test_matches_a_stable_sort(cuda_lib, n, values, dtype):
    gen = torch.Generator(device="cuda").manual_seed(n)
    ids = torch.randint(-(values // 2), values - values // 2, (n,), generator=gen, device="cuda").to(dtype)
    ordered, perm = torch.full((2, n + 1), -7, dtype=torch.int32, device="cuda")
    code = cuda_lib.lib().ctb_sort_ids(cuda_lib.ptr(ids), ids.element_size(), ctypes.c_long(n), cuda_lib.ptr(ordered),
                                       cuda_lib.ptr(perm), cuda_lib.stream_ptr())
    assert code == 0
    want = torch.sort(ids.to(torch.int32), stable=True)
    assert torch.equal(ordered[:n], want.values) and torch.equal(perm[:n].long(), want.indices)
    assert int(ordered[n]) == -7 and int(perm[n]) == -7


@pytest.mark.parametrize("n", [2048, 2049])
def test_embedding_gradient_of_both_sorts(cuda_lib, n):
    from causal_trainer_dev_b200.ops import elementwise as E

    gen = torch.Generator(device="cuda").manual_seed(3)
    ids = torch.randint(0, 300, (1, n), generator=gen, device="cuda")
    dout = torch.randn(n, 64, generator=gen, device="cuda").bfloat16()
    grad = torch.zeros(300, 64, device="cuda")
    E.embedding_backward(ids, dout, grad, pad_id=5)
    want = torch.zeros(300, 64, dtype=torch.float64, device="cuda").index_add_(0, ids[0], dout.double())
    want[5] = 0
    assert ((grad.double() - want).norm() / want.norm()).item() < 1e-5      # fp32 sums of some 50 rows
