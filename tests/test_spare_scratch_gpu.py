"""Scratch that a captured graph addresses is not replaced by a later, larger
call on the same engine: the call goes without, and the graph replays."""
import numpy as np
import pytest
import torch

from deepcharacters_b200 import synthetic as S
from deepcharacters_b200.renderer import RendererEngine, renderer_backward

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _t(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV)


def _captured(f):
    f()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = f()
    return g, out


def test_uv_maps_replay_after_a_larger_call():
    sc = S.render_scene(3, batch=5, views=1, width=40, height=32, seed=21, texture_size=37)
    eng = RendererEngine(sc["faces"], sc["texcoords"], sc["N"], 1, 40, 32, "vertexColor", "shadeless", 2, 2, "normal")
    args = [_t(sc["verts"]), _t(sc["colors"]), torch.zeros((5, 37, 37, 3), device=DEV), _t(sc["sh"]), _t(sc["extr"]),
            _t(sc["intr"])]
    one = [a[:1].contiguous() for a in args]
    g, got = _captured(lambda: eng.forward(*one))
    want = eng.forward(*args)[4]
    got[4].zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(got[4], want[:1])
    del g


def test_texture_gradient_replays_after_a_larger_texture():
    sc = S.render_scene(3, batch=1, views=1, width=64, height=64, seed=33, texture_size=16)
    eng = RendererEngine(sc["faces"], sc["texcoords"], sc["N"], 1, 64, 64, "textured", "shadeless", 2, 2)
    x = {k: _t(sc[k]) for k in ("verts", "colors", "texture", "sh", "target", "extr", "intr")}
    bary, face, render, vn, _ = eng.forward(x["verts"], x["colors"], x["texture"], x["sh"], x["extr"], x["intr"])
    grad = torch.randn(render.shape, device=DEV, generator=torch.Generator(DEV).manual_seed(4))
    run = lambda tex: renderer_backward(eng, grad, x["verts"], x["colors"], tex, x["sh"], x["target"], vn,  # noqa: E731
                                        bary, face, x["extr"], x["intr"])
    want = run(x["texture"])[2].clone()
    g, got = _captured(lambda: run(x["texture"]))
    large = run(torch.rand((1, 48, 48, 3), device=DEV))[2]
    got[2].zero_()
    g.replay()
    torch.cuda.synchronize()
    assert float(large.abs().sum()) > 0
    # FP32 sums in the order of the reductions
    assert float((got[2] - want).abs().max()) <= 1e-5 * float(want.abs().max())
    del g
