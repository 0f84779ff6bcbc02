"""Hinted boundary where triangles have many needed tiles: large triangles under a
poor hint, their boxes below and above the size that the warp shares."""
import numpy as np
import pytest
import torch

from deepcharacters_b200 import synthetic as S
from deepcharacters_b200.silhouette import MeshBoundaryEngine

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _scene(kind, res):
    rng = np.random.default_rng(3)
    if kind == "quad":  # a sphere in front of two triangles that span the view
        v, f = S.icosphere(5 if res < 1024 else 6)
        q = np.array([[-3000, -3000, 900], [3000, -3000, 900], [3000, 3000, 900], [-3000, 3000, 900.0]])
        v, f = np.concatenate([v * 600.0, q]), np.concatenate([f, np.array([[0, 1, 2], [0, 2, 3]]) + len(v)])
    else:
        m, size = 400, {"soup": 1500.0, "medium": 250.0}[kind]
        v = (rng.uniform(-1200, 1200, (m, 1, 3)) + rng.uniform(-size, size, (m, 3, 3))).reshape(-1, 3)
        f = np.arange(3 * m).reshape(-1, 3)
    k = res / 512 * 600.0
    extr = torch.tensor([[1, 0, 0, 0, 0, 1, 0, 0, 0, 0, 1, 3000.0]], device=DEV).reshape(1, 1, 3, 4)
    intr = torch.tensor([[k, 0, res / 2, 0, k, res / 2, 0, 0, 1]], device=DEV).reshape(1, 1, 3, 3)
    eng = MeshBoundaryEngine(f, len(v))
    verts = torch.from_numpy(np.ascontiguousarray(v[None], np.float32)).to(DEV)
    return lambda hint: eng.forward(verts, extr, intr, res, res, face_hint=hint), len(f)


@pytest.mark.parametrize("kind", ["quad", "soup", "medium"])
@pytest.mark.parametrize("res", [200, 517])
def test_flags_do_not_depend_on_the_hint(kind, res):
    run, n_faces = _scene(kind, res)
    want = run(None).clone()
    g = torch.Generator(DEV).manual_seed(1)
    for hint in (torch.full((1, 1, res, res), -1, dtype=torch.int32, device=DEV),
                 torch.randint(-1, n_faces, (1, 1, res, res), dtype=torch.int32, device=DEV, generator=g)):
        assert torch.equal(run(hint), want)


def test_poor_hint_costs_no_more_than_none():
    """Half of the unhinted time here; a thread alone on a large box takes three times."""
    res = 1024
    run, _ = _scene("quad", res)
    hint = torch.full((1, 1, res, res), -1, dtype=torch.int32, device=DEV)

    def best(h):
        ms = []
        for _ in range(10):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(5):
                run(h)
            b.record()
            b.synchronize()
            ms.append(a.elapsed_time(b))
        return min(ms)

    assert best(hint) < 1.5 * best(None)
