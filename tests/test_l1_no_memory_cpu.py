"""The image L1 where there is no memory for its scratch: the call without it."""
import pytest
import torch

from deepcharacters_b200 import losses as L


@pytest.mark.parametrize("room", [True, False])
def test_entry_point_by_memory(monkeypatch, room):
    calls = []
    empty = torch.empty

    def fake_empty(shape, **k):
        if k.get("dtype") is torch.uint8 and not room:
            raise torch.OutOfMemoryError("no memory")
        return empty(shape, **k)

    monkeypatch.setattr(L, "_f32", lambda t, name: t)
    monkeypatch.setattr(L, "_stream", lambda: 0)
    monkeypatch.setattr(L._lib, "call", lambda name, *a: calls.append((name, len(a))))
    monkeypatch.setattr(torch, "empty", fake_empty)
    loss, grad = L.image_l1_loss(torch.zeros((5, 3)), torch.zeros((5, 3)), torch.zeros(5, dtype=torch.int32))
    assert loss.shape == (1,) and grad.shape == (5, 3)
    name = "hc_image_l1_loss_scratch" if room else "hc_image_l1_loss"
    assert calls == [(name, len(L._lib._SIGS[name]))]
