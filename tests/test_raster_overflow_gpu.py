"""Triangles whose FP32 hit test overflows: the barycentrics of a pixel near an
edge are NaN, which no comparison of the window accepts, so the pixel stays
background (rayTriangleIntersect, CudaRenderer/cpp/src/Utils/RendererUtil.h:26-101)."""
import numpy as np
import pytest
import torch

from deepcharacters_b200.renderer import RendererEngine

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _faces(verts, face, tile):
    eng = RendererEngine(np.array(face, np.int32), None, 3, 1, 128, 128, "vertexColor", "shadeless", 2, 2)
    eng.set_tuning(tile, 512)
    extr = torch.eye(4, device=DEV)[:3].reshape(1, 1, 3, 4)
    intr = torch.tensor([[100.0, 0, 64, 0, 100, 64, 0, 0, 1]], device=DEV).reshape(1, 1, 3, 3)
    v = torch.from_numpy(np.asarray(verts, np.float32)[None]).to(DEV)
    return eng.forward(v, torch.ones((1, 3, 3), device=DEV), None, None, extr, intr)[1][0, 0].cpu().numpy()


@pytest.mark.parametrize("tile", [8, 16, 32])
@pytest.mark.parametrize("face", [[0, 1, 2], [0, 2, 1]])
def test_squared_normal_beyond_fp32(face, tile):
    # edges of 1e13 mm: |N|^2 is infinite, a pixel's numerators finite or infinite
    z = 1e13
    px = np.array([[40.4375, 10], [40.4375, 110], [100, 60]])
    f = _faces(np.stack([(px[:, 0] - 64) / 100 * z, (px[:, 1] - 64) / 100 * z, np.full(3, z)], 1), face, tile)
    assert (f[45:75, 40] == -1).all()  # pixel centres 0.0625 px inside the left edge
    assert (f[:, :40] == -1).all() and f[60, 60] == 0  # clearly inside: the depth alone decides
