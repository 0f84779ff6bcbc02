"""Tiles a triangle reaches, found row by row: wide, tall, thin and diagonal
triangles, boxes on both sides of a thread's share of tiles and of more than
32 rows, against the FP64 oracles."""
import numpy as np
import pytest
import torch

from deepcharacters_b200 import synthetic as S
from deepcharacters_b200.silhouette import MeshBoundaryEngine
from oracle import oracle as O
from oracle import silhouette_oracle as SO

from test_renderer_gpu import run_ours  # same directory

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("tile,cap", [(8, 512), (16, 512), (32, 1024), (8, 12)])
@pytest.mark.parametrize("subdiv,size,stretch", [(1, (340, 24), (4, 0.2, 1)), (1, (24, 340), (0.2, 4, 1)),
                                                 (2, (160, 160), (1, 1, 1)), (0, (600, 40), (6, 1, 1)),
                                                 (3, (130, 97), (1, 0.05, 1)), (3, (97, 130), (0.03, 1, 1))])
def test_faces_match_the_oracle(subdiv, size, stretch, tile, cap):
    W, H = size
    sc = S.render_scene(subdiv, batch=1, views=2, width=W, height=H, seed=21, fx=2.4 * min(W, H))
    rng = np.random.default_rng(9)
    v = sc["verts"] * np.float32(stretch)
    sc["verts"] = (v + rng.normal(0, 0.04 * np.abs(v).max(), v.shape)).astype(np.float32)  # diagonals
    ours = run_ours(sc, "vertexColor", "shadeless", tile, cap)
    ora = O.render_forward(sc["faces"], sc["texcoords"], 1, 2, W, H, "vertexColor", "shadeless", sc["verts"],
                           sc["colors"], sc["texture"], sc["sh"], sc["extr"], sc["intr"])
    robust = (ora["fragile"] == 0) & (ora["tie_count"] < 2) & (ours["tie_count"] < 2)
    assert np.array_equal(ours["face"][robust], ora["face"][robust])
    assert (robust & (ora["face"] >= 0)).any()


@pytest.mark.parametrize("size", [(300, 20), (20, 300), (140, 130)])
@pytest.mark.parametrize("extent", [(200.0, 3.0), (3.0, 200.0), (30.0, 30.0), (90.0, 90.0)])
def test_flags_match_the_oracle(size, extent):
    W, H = size
    rng = np.random.default_rng(W + int(extent[0]))
    count = 25
    centre = rng.uniform(0, 1, size=(count, 1, 2)) * [W, H]
    tri = (centre + rng.uniform(-1, 1, size=(count, 3, 2)) * extent).reshape(-1, 2)
    x, y = np.meshgrid(np.arange(1, W - 1, 2) + 0.3, np.arange(1, H - 1, 2) + 0.6)
    p2d = np.concatenate([tri, np.stack([x.ravel(), y.ravel()], 1)]).astype(np.float32)[None, None]
    faces = np.arange(3 * count, dtype=np.int32).reshape(-1, 3)
    N = p2d.shape[2]
    eng = MeshBoundaryEngine(faces, N)
    zeros, ex, it = (torch.zeros(s, device=DEV) for s in ((1, N, 3), (1, 12), (1, 9)))
    ours = eng.forward(zeros, ex, it, W, H, points_image_space=torch.from_numpy(p2d).to(DEV))
    # FP64 differs only where a pixel centre sits on the barycentric tolerance
    assert int((ours.cpu().numpy() != SO.mesh_boundary(faces, p2d, W, H)).sum()) <= 2
