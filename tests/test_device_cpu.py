"""Host-side parts of the device layer that need no GPU."""
import torch

from tenex_b200.kernels import device as D


def test_to_device_takes_a_tensor_that_requires_grad():
    x = torch.arange(6, dtype=torch.float32).reshape(2, 3)
    got = D.to_device(x.clone().requires_grad_(), "cpu")
    assert torch.equal(got, x)
