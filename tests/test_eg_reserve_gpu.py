"""hc_eg_reserve takes the full skinned gradient's memory where that gradient is on,
before or after the call, and no more without it."""
import numpy as np
import pytest
import torch

from deepcharacters_b200 import _lib
from deepcharacters_b200.embedded_graph import EGData, EmbeddedGraphEngine

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _engine(n, m, full):
    rng = np.random.default_rng(n)
    base = rng.normal(0, 500.0, size=(n, 3)).astype(np.float32)
    faces = np.stack([rng.permutation(n)[:3] for _ in range(2 * n)]).astype(np.int32)
    vid = np.arange(n, dtype=np.int32)
    idx = (vid % m).astype(np.int32)
    order = np.lexsort((vid, idx))
    sizes = np.bincount(idx, minlength=m).astype(np.int32)
    w = np.ones(n, np.float32)
    return EmbeddedGraphEngine(EGData(base, faces, rng.permutation(n)[:m].astype(np.int32), vid,
                                      np.ones(n, np.int32), idx, w,
                                      np.concatenate([[0], np.cumsum(sizes)[:-1]]).astype(np.int32), sizes, vid[order],
                                      w, None, None), full_skinned_gradient=full)


def test_memory_without_the_full_gradient():
    eng = _engine(2000, 4, False)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    eng.reserve(5000)  # the packed vertices would take 480 MB
    assert before - torch.cuda.mem_get_info()[0] < 64 << 20


@pytest.mark.parametrize("late", [False, True])
def test_captured_after_reserve(late):
    B, n, m = 3, 300, 20
    eng = _engine(n, m, not late)
    eng.reserve(B)
    if late:  # the full gradient switched on after the reservation
        _lib.call("hc_eg_set_full_skinned_gradient", eng.handle, 1)
        eng.full = True
    g = torch.Generator(DEV).manual_seed(2)
    f = lambda s, *shape: torch.randn(shape, device=DEV, generator=g) * s  # noqa: E731
    x = [f(10.0, B, m, 3), f(0.3, B, m, 3), f(20.0, B, m, 3), f(0.4, B, m, 3), f(1.0, B, n, 3)]
    gv = f(1.0, B, n, 3)
    other = _engine(n, m, True)
    da, sa = other.forward(*x)[4:]
    want = other.backward(gv, None, da, sa, x[0], x[4])
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):  # the first call on this engine
        da, sa = eng.forward(*x)[4:]
        got = eng.backward(gv, None, da, sa, x[0], x[4])
    graph.replay()
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        assert torch.equal(a, b) and float(b.abs().sum()) > 0
