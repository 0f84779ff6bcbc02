"""The embedded graph's adjoint without skinned gradients beyond the grid's 65,535
frames: the same values as in two calls."""
import numpy as np
import pytest
import torch

from deepcharacters_b200.embedded_graph import EGData, EmbeddedGraphEngine

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("frames", [65535, 65536, 70000])
def test_adjoint_of_many_frames(frames):
    n, m = 7, 2
    rng = np.random.default_rng(1)
    base = rng.normal(0, 500.0, size=(n, 3)).astype(np.float32)
    faces = np.array([[0, 1, 2], [2, 3, 4], [4, 5, 6]], np.int32)
    vid, idx = np.arange(n, dtype=np.int32), (np.arange(n) % m).astype(np.int32)
    order = np.lexsort((vid, idx))
    w = np.ones(n, np.float32)
    eng = EmbeddedGraphEngine(EGData(base, faces, np.array([0, 3], np.int32), vid, np.ones(n, np.int32), idx, w,
                                     np.array([0, 4], np.int32), np.array([4, 3], np.int32), vid[order], w, None, None))
    g = torch.Generator(DEV).manual_seed(2)
    gv = torch.randn((frames, n, 3), device=DEV, generator=g)
    da, sa = (0.3 * torch.randn((frames, m, 3), device=DEV, generator=g) for _ in range(2))
    got = eng.backward(gv, None, da, sa)
    parts = [eng.backward(gv[a:b], None, da[a:b], sa[a:b]) for a, b in ((0, 40000), (40000, frames))]
    for t, *p in zip(got, *parts):
        assert torch.equal(t, torch.cat(p))
    assert float(got[4][-1].abs().sum()) > 0
