"""The silhouette's per-pixel passes at the edges of their 4096-pixel blocks,
with 16-byte words and without, dense and sparse contours, against the FP64
oracle."""
import numpy as np
import pytest
import torch

from deepcharacters_b200 import synthetic as S
from deepcharacters_b200.silhouette import SilhouetteEngine, silhouette_backward
from oracle import silhouette_oracle as SO

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def nrel(a, b):
    a, b = a.double().cpu().numpy(), np.asarray(b, np.float64)
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30))


@pytest.mark.parametrize("U,V", [(64, 64), (68, 64), (65, 63), (12, 10), (128, 97), (63, 4)])
@pytest.mark.parametrize("dense", [False, True])
def test_blocks_match_the_oracle(U, V, dense):
    rng = np.random.default_rng(U * V)
    B, C, N = 1, 2, 150
    dt = S.silhouette_masks(B, C, U, V, seed=3, scale=min(U, V) / 512.0)  # [B,C,V,U]
    if dense:  # every pixel of some rows on the contour
        dt[:, :, V // 2:V // 2 + 3] = 127
    # points on a grid of quarter pixels with distinct distances almost surely
    p2d = (rng.uniform(0, 1, size=(B, C, N, 2)) * [U, V]).astype(np.float32)
    n2d = rng.normal(size=(B, C, N, 2)).astype(np.float32)
    n2d /= np.linalg.norm(n2d, axis=-1, keepdims=True)
    isb = (rng.random((B, C, N)) < 0.5).astype(np.uint8)
    crops = S.identity_crops(B, C, U, V)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)  # noqa: E731
    d4 = dt.reshape(B, C, U, V)  # the op's [B,C,U,V] naming of the same memory
    ours = SilhouetteEngine().forward(t(p2d), t(n2d), t(isb), t(d4), t(crops))
    ora = SO.silhouette_forward(p2d, n2d, isb, d4, crops)
    assert np.array_equal(ours[3].cpu().numpy(), ora[3])
    assert nrel(ours[1], ora[1]) < 1e-6
    g, g1 = rng.normal(size=(B, C, N)).astype(np.float32), rng.normal(size=ora[1].shape).astype(np.float32)
    out = silhouette_backward(t(g), t(g1), ours[2], ours[3], t(crops))
    assert nrel(out, SO.silhouette_backward(g, g1, ours[2].double().cpu().numpy(), ora[3], crops)) < 1e-6
