"""The needed-tile words of the hinted boundary: images whose tile rows and
columns end inside, at and just past a word, mixed sizes, against the unhinted
flags."""
import numpy as np
import pytest
import torch

from deepcharacters_b200 import synthetic as S
from deepcharacters_b200.silhouette import MeshBoundaryEngine

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("sizes", [[(64, 64)] * 3, [(65, 64)] * 2, [(57, 129)] * 2, [(520, 40), (72, 72), (9, 300)]])
def test_hinted_flags_equal_the_full_ones(sizes):
    C, B = len(sizes), 2
    w, h = ([s[k] for s in sizes] for k in (0, 1))
    sc = S.render_scene(4, batch=B, views=C, width=64, height=64, seed=3)
    it = np.concatenate([S.camera_ring(1, 3000.0, 0.5 * min(s) + 8.0, *s)[1] for s in sizes])
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)  # noqa: E731
    verts, ex, it = t(sc["verts"]), t(sc["extr"]), t(np.tile(it[None], (B, 1)))
    eng = MeshBoundaryEngine(sc["faces"], sc["N"])
    full = eng.forward_sized(verts, ex, it, w, h).clone()
    assert 0 < int(full.sum()) < full.numel()
    P = sum(a * b for a, b in sizes)
    g = torch.Generator(DEV).manual_seed(1)
    for hint in (torch.full((B, P), -1, dtype=torch.int32, device=DEV),
                 torch.randint(-1, len(sc["faces"]), (B, P), generator=g, device=DEV, dtype=torch.int32)):
        assert torch.equal(eng.forward_sized(verts, ex, it, w, h, face_hint=hint), full)
