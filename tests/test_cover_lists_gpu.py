"""Per-pixel lists of the coverage tiles: triangle soups that leave remainders
of 32 and 64 records in a tile, on images that cut tiles, against the FP64
oracle; with and without a hint."""
import numpy as np
import pytest
import torch

from deepcharacters_b200.silhouette import MeshBoundaryEngine
from oracle import silhouette_oracle as SO

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("size", [(9, 11), (37, 23), (64, 40)])
@pytest.mark.parametrize("count,extent", [(20, 3.0), (33, 6.0), (70, 12.0), (230, 2.0), (40, 60.0)])
def test_flags_match_the_oracle(size, count, extent):
    W, H = size
    rng = np.random.default_rng(count * W)
    centre = rng.uniform(0, 1, size=(count, 1, 2)) * [W, H]
    tri = (centre + rng.uniform(-extent, extent, size=(count, 3, 2))).reshape(-1, 2)
    x, y = np.meshgrid(np.arange(1, W - 1, 2) + 0.3, np.arange(1, H - 1, 2) + 0.6)
    p2d = np.concatenate([tri, np.stack([x.ravel(), y.ravel()], 1)]).astype(np.float32)[None, None]
    faces = np.arange(3 * count, dtype=np.int32).reshape(-1, 3)
    N = p2d.shape[2]
    eng = MeshBoundaryEngine(faces, N)
    zeros, ex, it = (torch.zeros(s, device=DEV) for s in ((1, N, 3), (1, 12), (1, 9)))
    pts = torch.from_numpy(p2d).to(DEV)
    ours = eng.forward(zeros, ex, it, W, H, points_image_space=pts).clone()
    hint = torch.full((1, 1, H, W), -1, dtype=torch.int32, device=DEV)
    assert torch.equal(ours, eng.forward(zeros, ex, it, W, H, points_image_space=pts, face_hint=hint))
    # FP64 differs only where a pixel centre sits on the barycentric tolerance
    assert int((ours.cpu().numpy() != SO.mesh_boundary(faces, p2d, W, H)).sum()) <= 2
