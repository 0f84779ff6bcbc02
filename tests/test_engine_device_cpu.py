"""Cached renderer engines belong to a device: another device's calls get their own,
made and run with that device current, and tensors elsewhere are refused.  The
devices are stood in for on the host."""
import contextlib
import types

import numpy as np
import pytest
import torch

from deepcharacters_b200 import renderer as R


@pytest.fixture
def devices(monkeypatch):
    state = types.SimpleNamespace(current=0)

    @contextlib.contextmanager
    def device(i):
        before, state.current = state.current, i
        yield
        state.current = before

    class Engine:
        def __init__(self, *a):
            self.device = state.current

    monkeypatch.setattr(torch.cuda, "current_device", lambda: state.current)
    monkeypatch.setattr(torch.cuda, "device", device)
    monkeypatch.setattr(R, "RendererEngine", Engine)
    monkeypatch.setattr(R, "_ENGINES", [])
    return state


def _get(device=None, width=32):
    return R.get_engine(np.array([0, 1, 2], np.int32), None, 3, 1, width, 32, "vertexColor", "shadeless", 2, 2,
                        "none", *([] if device is None else [device]))


def test_engines_of_two_devices(devices):
    a, b = _get(0), _get(1)
    assert a is not b and (a.device, b.device) == (0, 1) and devices.current == 0
    assert _get(0) is a is _get() and _get(1) is b
    devices.current = 1
    assert _get() is b
    for k in range(R._ENGINES_MOST + 3):  # one device's engines do not push out another's
        _get(0, 40 + k)
    assert _get(1) is b and _get(0) is not a
    assert [e[0][-1] for e in R._ENGINES].count(0) == R._ENGINES_MOST


def test_tensors_on_another_device_are_refused(monkeypatch):
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: types.SimpleNamespace(device_index=0, cuda_stream=0))
    eng = object.__new__(R.RendererEngine)
    eng.device = 1
    v = types.SimpleNamespace(is_cuda=True, dtype=torch.float32, is_contiguous=lambda: True, shape=(1, 3, 3),
                              device=torch.device("cuda", 0))
    with pytest.raises(ValueError, match="vertex_pos is on cuda:0, the engine on cuda:1"):
        eng.forward(v, None, None, None, None, None)
    with pytest.raises(ValueError, match="vertex_pos is on cuda:0, the engine on cuda:1"):
        R.renderer_backward(eng, None, v, *[None] * 9)
