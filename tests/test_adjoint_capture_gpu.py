"""The adjoint's per-vertex sums follow the cameras' buffer: a larger backward can be
captured after a larger forward, and a captured backward outlives a larger one."""
import numpy as np
import pytest
import torch

from deepcharacters_b200 import synthetic as S
from deepcharacters_b200.renderer import RendererEngine, renderer_backward

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _setup(shading):
    sc = S.render_scene(3, batch=4, views=2, width=48, height=40, seed=33, texture_size=16)
    x = {k: torch.from_numpy(np.ascontiguousarray(sc[k])).to(DEV)
         for k in ("verts", "colors", "texture", "sh", "target", "extr", "intr")}
    make = lambda: RendererEngine(sc["faces"], sc["texcoords"], sc["N"], 2, 48, 40, "vertexColor", shading, 2, 2)  # noqa: E731

    def forward(eng, b):
        y = {k: t[:b].contiguous() for k, t in x.items()}
        return y, eng.forward(y["verts"], y["colors"], y["texture"], y["sh"], y["extr"], y["intr"])

    def backward(eng, y, o):
        return renderer_backward(eng, torch.ones_like(o[2]), y["verts"], y["colors"], y["texture"], y["sh"],
                                 y["target"], o[3], o[0], o[1], y["extr"], y["intr"])

    return make, forward, backward


def _same(got, want):
    for a, b in zip(got, want):  # FP32 sums in the order of the reductions
        assert float((a - b).abs().max()) <= 1e-5 * max(float(b.abs().max()), 1e-30)


def _graph(f):
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = f()
    return g, out


def test_capture_of_a_larger_backward():
    make, forward, backward = _setup("shadeless")
    want = backward(make(), *forward(make(), 4))
    eng = make()
    backward(eng, *forward(eng, 1))
    forward(eng, 4)
    g, got = _graph(lambda: backward(eng, *forward(eng, 4)))
    g.replay()
    torch.cuda.synchronize()
    _same(got, want)


@pytest.mark.parametrize("shading", ["shadeless", "shaded"])
def test_captured_backward_after_a_larger_one(shading):
    make, forward, backward = _setup(shading)
    eng = make()
    forward(eng, 4)
    eng.set_tuning(32, 512)
    y, o = forward(eng, 1)
    want = [t.clone() for t in backward(eng, y, o)]
    g, got = _graph(lambda: backward(eng, y, o))
    backward(eng, *forward(eng, 4))
    for t in got:
        t.fill_(7.0)
    g.replay()
    torch.cuda.synchronize()
    _same(got, want)


def test_capture_after_reserve_alone():
    make, forward, backward = _setup("shaded")
    want = backward(make(), *forward(make(), 4))  # loads the kernels too
    eng = make()
    eng.reserve(4)
    g, got = _graph(lambda: backward(eng, *forward(eng, 4)))
    g.replay()
    torch.cuda.synchronize()
    _same(got, want)
