"""Captured textured adjoints after larger eager ones, where both want the padded
texel sums (at least two pixels per texel, bilinear) or the padded texture."""
import numpy as np
import pytest
import torch

from deepcharacters_b200 import synthetic as S
from deepcharacters_b200.renderer import RendererEngine, renderer_backward

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("albedo,small,large", [("texturedBilinear", 16, 40), ("textured", 8, 16)])
def test_texture_gradient_replays(albedo, small, large):
    # 4096 pixels: the sums are padded for up to 2048 texels bilinear, 256 nearest
    sc = S.render_scene(3, batch=1, views=1, width=64, height=64, seed=33, texture_size=small)
    eng = RendererEngine(sc["faces"], sc["texcoords"], sc["N"], 1, 64, 64, albedo, "shadeless", 2, 2)
    x = {k: torch.from_numpy(np.ascontiguousarray(sc[k])).to(DEV)
         for k in ("verts", "colors", "texture", "sh", "target", "extr", "intr")}
    bary, face, render, vn, _ = eng.forward(x["verts"], x["colors"], x["texture"], x["sh"], x["extr"], x["intr"])
    grad = torch.randn(render.shape, device=DEV, generator=torch.Generator(DEV).manual_seed(4))

    def run(tex):
        return renderer_backward(eng, grad, x["verts"], x["colors"], tex, x["sh"], x["target"], vn, bary, face,
                                 x["extr"], x["intr"])[2]

    big = torch.rand((1, large, large, 3), device=DEV)
    want = run(x["texture"]).clone()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        got = run(x["texture"])
    first = run(big).clone()  # without the padded buffers, which the graph holds
    got.zero_()
    g.replay()
    torch.cuda.synchronize()
    # FP32 sums in the order of the reductions
    assert float((got - want).abs().max()) <= 1e-5 * float(want.abs().max())
    other = RendererEngine(sc["faces"], sc["texcoords"], sc["N"], 1, 64, 64, albedo, "shadeless", 2, 2)
    eng = other  # with them
    assert float((run(big) - first).abs().max()) <= 1e-5 * float(first.abs().max())
