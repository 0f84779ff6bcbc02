"""The adjoint's per-vertex sums and texture taps against the FP64 oracle, for
every number of values per vertex (shading x albedo), with the target staged
by TMA (rows of 16-byte multiples) and without, on images that cut tiles."""
import numpy as np
import pytest
import torch

from deepcharacters_b200 import synthetic as S
from deepcharacters_b200.renderer import RendererEngine, renderer_backward
from oracle import oracle as O

from _conditioning import well_conditioned_mask

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TOL = 1e-5  # norm-wise relative, FP32: the bar of the adjoint against the FP64 oracle


def _t(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV)


def nrel(a, b):
    a, b = a.double().cpu(), torch.from_numpy(b).double()
    return float((a - b).norm() / max(b.norm().item(), 1e-30))


@pytest.mark.parametrize("parity", [False, True])
@pytest.mark.parametrize("albedo,shading,tfs", [("vertexColor", "shadeless", 2), ("vertexColor", "shaded", 2),
                                                ("textured", "shadeless", 1), ("textured", "shaded", 2),
                                                ("textured", "shaded", 3), ("textured", "shadeless", 5)])
@pytest.mark.parametrize("size", [(100, 52), (75, 43)])
def test_sums_match_the_oracle(size, albedo, shading, tfs, parity):
    W, H = size
    sc = S.render_scene(3, batch=2, views=2, width=W, height=H, seed=31, texture_size=96)
    eng = RendererEngine(sc["faces"], sc["texcoords"], sc["N"], 2, W, H, albedo, shading, 2, tfs)
    eng.set_gradient_parity(parity)
    x = {k: _t(sc[k]) for k in ("verts", "colors", "texture", "sh", "target", "extr", "intr")}
    bary, face, render, vn, _ = eng.forward(x["verts"], x["colors"], x["texture"], x["sh"], x["extr"], x["intr"])
    keep = well_conditioned_mask(sc["verts"], sc["faces"], sc["texcoords"], 96, sc["extr"], sc["intr"],
                                 face.cpu().numpy(), bary.cpu().numpy(), albedo)
    g = torch.randn(render.shape, device=DEV, generator=torch.Generator(DEV).manual_seed(4)) * _t(keep[..., None])
    gpos, gcol, gtex, gsh = renderer_backward(eng, g, x["verts"], x["colors"], x["texture"], x["sh"], x["target"], vn,
                                              bary, face, x["extr"], x["intr"])
    args = (sc["faces"], sc["texcoords"], 2, 2, W, H, albedo, shading, g.cpu().numpy(), sc["verts"], sc["colors"],
            sc["texture"], sc["sh"], sc["target"], vn.cpu().numpy(), bary.cpu().numpy(), face.cpu().numpy(),
            sc["extr"], sc["intr"])
    o64, o32 = (O.render_backward(*args, ifs=2, tfs=tfs, precision=p) for p in ("f64", "f32"))
    assert keep.any() and float(gpos.abs().max()) > 0
    pairs = [(gpos, "vertex_pos_grad")]
    pairs += [(gcol, "vertex_color_grad")] if albedo == "vertexColor" else [(gtex, "texture_grad")]
    pairs += [(gsh, "sh_coeff_grad")] if shading == "shaded" else []
    for ours, key in pairs:
        # no further than the reference formula evaluated in FP32, or the FP32 bar
        floor = nrel(torch.from_numpy(o32[key]), o64[key])
        assert nrel(ours, o64[key]) < max(TOL, 1.25 * floor), (key, nrel(ours, o64[key]), floor)
    if albedo != "vertexColor":
        assert float(gcol.abs().max()) == 0.0
    if shading != "shaded":
        assert float(gsh.abs().max()) == 0.0
