"""The renderer wrapper's engine lookup goes by contents, and gradients that no
input asks for are left out."""
import numpy as np
import pytest
import torch

from deepcharacters_b200 import renderer as R
from deepcharacters_b200 import synthetic as S

pytestmark = pytest.mark.gpu


def test_engines_are_found_by_contents():
    sc = S.render_scene(2, batch=1, views=1, width=32, height=32, seed=1)
    f, tc = sc["faces"].copy(), sc["texcoords"].copy()
    rest = (sc["N"], 1, 32, 32, "vertexColor", "shadeless", 2, 2, "none")
    a = R.get_engine(f, tc, *rest)
    assert R.get_engine(f.copy(), tc.copy(), *rest) is a
    assert R.get_engine(f.reshape(-1).tolist(), tc.tolist(), *rest) is a
    assert R.get_engine(f, None, *rest) is not a and R.get_engine(f, tc, *rest[:-3], 1, *rest[-2:]) is not a
    f[[0, 1]] = f[[1, 0]]  # the same array with other contents is another mesh
    b = R.get_engine(f, tc, *rest)
    assert b is not a and R.get_engine(sc["faces"], sc["texcoords"], *rest) is a
    tc[0] = np.nan  # compared as bytes
    assert R.get_engine(f, tc, *rest) is R.get_engine(f, tc.copy(), *rest)
    for k in range(R._ENGINES_MOST + 3):
        R.get_engine(f, None, sc["N"], 1, 33 + k, 32, *rest[4:])
    assert len(R._ENGINES) == R._ENGINES_MOST


@pytest.mark.parametrize("asked", [False, True])
def test_target_and_camera_gradients(asked):
    sc = S.render_scene(2, batch=1, views=1, width=32, height=32, seed=1)
    t = lambda k, g=False: torch.from_numpy(sc[k]).cuda().requires_grad_(g)  # noqa: E731
    x = [t("verts", True), t("colors", True), t("texture", True), t("sh", True), t("target", asked),
         t("extr", asked), t("intr", asked)]
    r = R.CudaRendererGpu(sc["faces"], sc["texcoords"], sc["N"], 1, 32, 32, "vertexColor", "shadeless", 2, 2, "none",
                          *x)
    r.getRenderBufferTF().sum().backward()
    assert float(x[1].grad.abs().sum()) > 0 and float(x[2].grad.abs().max()) == 0 == float(x[3].grad.abs().max())
    for k in x[4:]:
        assert (k.grad is not None and float(k.grad.abs().max()) == 0) if asked else k.grad is None
    # a loss on another output alone leaves the renderer's gradients at zero
    r = R.CudaRendererGpu(sc["faces"], sc["texcoords"], sc["N"], 1, 32, 32, "vertexColor", "shadeless", 2, 2, "none",
                          *x)
    g = torch.autograd.grad(r.getVertexNormalTF().sum(), x[:2])
    assert all(float(v.abs().max()) == 0 for v in g)
