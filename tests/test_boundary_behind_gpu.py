"""Boundary flags with vertices behind the camera, whose projections pass 2^31 pixels:
they have no window in the image and are not on the boundary, and the others' flags
are those of a mesh that ends before them."""
import numpy as np
import pytest
import torch

from deepcharacters_b200 import synthetic as S
from deepcharacters_b200.silhouette import (MeshBoundaryEngine, camera_projection_forward, projected_mesh_boundary)

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("res", [33, 160])
def test_vertices_behind_the_camera(res):
    v, f = S.icosphere(3)
    n = len(v)
    # right behind the camera's plane, so that either sign occurs
    v = np.concatenate([v * 700.0, np.random.default_rng(1).uniform(-900, 900, (300, 3)) * [1, 1, 0.05] - [0, 0, 3050]])
    extr = torch.tensor([[1, 0, 0, 0, 0, 1, 0, 0, 0, 0, 1, 3000.0]], device=DEV).reshape(1, 1, 3, 4)
    k = res / 512 * 600.0
    intr = torch.tensor([[k, 0, res / 2, 0, k, res / 2, 0, 0, 1]], device=DEV).reshape(1, 1, 3, 3)
    verts = torch.from_numpy(np.ascontiguousarray(v[None], np.float32)).to(DEV)
    p2d = camera_projection_forward(verts, None, extr, intr, 1)
    assert int((p2d[0, 0, n:] > 2.0 ** 31).all(-1).sum()) > 5  # both coordinates, by the z of 1e-5 behind the camera
    eng, front = MeshBoundaryEngine(f, len(v)), MeshBoundaryEngine(f, n)
    want = front.forward(verts[:, :n].contiguous(), extr, intr, res, res)
    assert 0 < int(want.sum()) < n
    g = torch.Generator(DEV).manual_seed(3)
    empty = torch.full((1, 1, res, res), -1, dtype=torch.int32, device=DEV)
    for hint in (None, empty, torch.randint(-1, len(f), empty.shape, dtype=torch.int32, device=DEV, generator=g)):
        flags = eng.forward(verts, extr, intr, res, res, face_hint=hint)
        assert torch.equal(flags[..., :n], want) and int(flags[..., n:].sum()) == 0
    flags = projected_mesh_boundary(p2d, empty, res, res)  # every pixel open
    inside = ((p2d >= 1) & (p2d < res - 1)).all(-1)
    assert torch.equal(flags != 0, inside) and int(flags[..., n:].sum()) == 0
