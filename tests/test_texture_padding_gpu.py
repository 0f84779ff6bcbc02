"""The adjoint with and without padded texels (chosen by pixels per texel):
nearest gradients against the FP64 oracle on both sides of the rule, bilinear
ones between the two sides on the same pixels."""
import numpy as np
import pytest
import torch

from deepcharacters_b200 import synthetic as S
from deepcharacters_b200.renderer import RendererEngine, renderer_backward
from oracle import oracle as O

from _conditioning import well_conditioned_mask
from test_vertex_sums_gpu import TOL, _t, nrel  # same directory

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tfs", [1, 2, 3])
@pytest.mark.parametrize("size,texture", [(40, 97), (60, 13), (64, 64)])
def test_nearest_texels_match_the_oracle(size, texture, tfs):
    sc = S.render_scene(3, batch=1, views=2, width=size, height=size, seed=33, texture_size=texture)
    eng = RendererEngine(sc["faces"], sc["texcoords"], sc["N"], 2, size, size, "textured", "shaded", 2, tfs)
    x = {k: _t(sc[k]) for k in ("verts", "colors", "texture", "sh", "target", "extr", "intr")}
    bary, face, render, vn, _ = eng.forward(x["verts"], x["colors"], x["texture"], x["sh"], x["extr"], x["intr"])
    keep = well_conditioned_mask(sc["verts"], sc["faces"], sc["texcoords"], texture, sc["extr"], sc["intr"],
                                 face.cpu().numpy(), bary.cpu().numpy(), "textured")
    g = torch.randn(render.shape, device="cuda:0", generator=torch.Generator("cuda:0").manual_seed(4))
    g = g * _t(keep[..., None])
    gpos, _, gtex, gsh = renderer_backward(eng, g, x["verts"], x["colors"], x["texture"], x["sh"], x["target"], vn,
                                           bary, face, x["extr"], x["intr"])
    args = (sc["faces"], sc["texcoords"], 1, 2, size, size, "textured", "shaded", g.cpu().numpy(), sc["verts"],
            sc["colors"], sc["texture"], sc["sh"], sc["target"], vn.cpu().numpy(), bary.cpu().numpy(),
            face.cpu().numpy(), sc["extr"], sc["intr"])
    o64, o32 = (O.render_backward(*args, ifs=2, tfs=tfs, precision=p) for p in ("f64", "f32"))
    for ours, key in ((gpos, "vertex_pos_grad"), (gtex, "texture_grad"), (gsh, "sh_coeff_grad")):
        floor = nrel(torch.from_numpy(o32[key]), o64[key])
        assert nrel(ours, o64[key]) < max(TOL, 1.25 * floor), (key, nrel(ours, o64[key]), floor)


def test_bilinear_sums_agree_on_both_sides_of_the_rule():
    """One view of a frame (in place) and the same view rendered four times (padded): four times the gradient."""
    sc = S.render_scene(3, batch=1, views=1, width=72, height=60, seed=3, texture_size=64)
    x = {k: _t(sc[k]) for k in ("verts", "colors", "texture")}
    g = torch.randn((1, 1, 60, 72, 3), device="cuda:0", generator=torch.Generator("cuda:0").manual_seed(4))
    out = []
    for C in (1, 4):
        ex, it, sh = (_t(np.tile(sc[k].reshape(1, -1), (1, C))) for k in ("extr", "intr", "sh"))
        eng = RendererEngine(sc["faces"], sc["texcoords"], sc["N"], C, 72, 60, "texturedBilinear", "shadeless", 2, 2)
        bary, face, render, vn, _ = eng.forward(x["verts"], x["colors"], x["texture"], sh.view(1, C, 27), ex, it)
        gc = g.expand(1, C, 60, 72, 3)
        out.append(renderer_backward(eng, gc, x["verts"], x["colors"], x["texture"], sh.view(1, C, 27),
                                     torch.zeros_like(render), vn, bary, face, ex, it))
    for k in (0, 2):  # positions, texture: FP32 sums in another order
        assert nrel(out[1][k], 4.0 * out[0][k].double().cpu().numpy()) < 1e-5
