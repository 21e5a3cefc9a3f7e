"""The factor of the loss gradients, as a number, a tensor on the host or one on the device."""
import pytest
import torch


@pytest.mark.parametrize("shape", [(), (1,), (1, 1)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, torch.bfloat16])
def test_a_tensor_on_the_host_becomes_a_number(shape, dtype):
    from causal_trainer_dev_b200.ops.cross_entropy import _device_scale

    scale = torch.full(shape, 0.37, dtype=dtype)
    number, on_device = _device_scale(scale, torch.device("meta"))       # (nothing may be moved there)
    assert on_device is None and number == float(scale.float())


def test_numbers_and_device_tensors():
    from causal_trainer_dev_b200.ops.cross_entropy import _device_scale

    assert _device_scale(0.5, torch.device("meta")) == (0.5, None)
    number, on_device = _device_scale(torch.empty(1, dtype=torch.float64, device="meta"), torch.device("meta"))
    assert number == 1.0 and on_device.shape == () and on_device.dtype == torch.float32
