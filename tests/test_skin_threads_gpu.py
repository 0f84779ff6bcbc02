"""Skinning handles whose blocks need different amounts of shared memory, used by
several threads at once: every launch is accepted and gives its handle's values."""
import ctypes
import threading

import numpy as np
import pytest
import torch

from deepcharacters_b200 import _lib
from deepcharacters_b200.skinning import Character, SkinningEngine

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _adjoint(k):
    """An engine with k slots per vertex and its prepared adjoint call."""
    rng = np.random.default_rng(k)
    n, s = 512, 9
    v = rng.normal(0, 100, (n, 3)).astype(np.float32)
    eng = SkinningEngine(Character(np.arange(-1, s - 1, dtype=np.int32), np.zeros(s, np.int32), np.ones((s, 3)),
                                   np.tile([[0, 0, 1.0]], (s, 1)), np.arange(s + 1), np.arange(s), np.ones(s),
                                   np.arange(s), v, v / 100, rng.integers(0, s, (n, k))))
    w = torch.full((1, n, k), 1.0 / k, device=DEV)
    o = eng.dq_forward(torch.full((1, s), 0.1, device=DEV), w)
    ins = [torch.ones((1, n, 3), device=DEV), o[0], o[2], o[3], o[4], w]
    out = [torch.zeros((1, s), device=DEV), torch.zeros((1, n, k), device=DEV)]
    stream = torch.cuda.Stream()
    args = [eng.handle, ctypes.c_void_p(stream.cuda_stream), 1] + [ctypes.c_void_p(t.data_ptr()) for t in ins + out]
    return eng, ins, out, stream, args


def test_handles_of_different_size_in_two_threads():
    fn = _lib.lib().hc_dq_skinning_backward
    calls = [_adjoint(44), _adjoint(24)]  # 94 and 54 KB of shared memory per block
    torch.cuda.synchronize()
    want = [eng.dq_backward(*ins)[1].clone() for eng, ins, *_ in calls]
    torch.cuda.synchronize()
    status = [set(), set()]

    def loop(i):
        args, stream = calls[i][4], calls[i][3]
        for k in range(6000):
            status[i].add(fn(*args))
            if k % 100 == 0:
                stream.synchronize()

    threads = [threading.Thread(target=loop, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert status == [{0}, {0}]
    for (_, _, out, *_), w in zip(calls, want):
        assert torch.equal(out[1], w)
