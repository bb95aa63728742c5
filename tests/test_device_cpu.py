"""Host-side parts of the device layer that need no GPU."""
import pytest
import torch

from tenex_b200 import native
from tenex_b200.kernels import device as D


def test_to_device_takes_a_tensor_that_requires_grad():
    x = torch.arange(6, dtype=torch.float32).reshape(2, 3)
    got = D.to_device(x.clone().requires_grad_(), "cpu")
    assert torch.equal(got, x)


def test_workspace_falls_back_to_the_least_when_memory_is_short(monkeypatch):
    L = native.lib()
    full = L.tenex_te_workspace_bytes(200, 3000, 16)
    least = L.tenex_te_pairs_workspace_bytes(200, 3000, 16)
    assert full > least
    real, asked = torch.empty, []

    def empty(nb, **kw):
        asked.append(nb)
        if nb > least:
            raise torch.OutOfMemoryError("no room")
        return real(nb, **kw)

    monkeypatch.setattr(torch, "empty", empty)
    assert D.workspace("cpu", 200, 3000, 16).numel() == least and asked == [full, least]
    monkeypatch.setattr(torch, "empty", lambda *a, **k: (_ for _ in ()).throw(
        torch.OutOfMemoryError("no room")))
    with pytest.raises(torch.OutOfMemoryError):
        D.workspace("cpu", 200, 3000, 16)
