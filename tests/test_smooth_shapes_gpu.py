"""Gaussian smoothing at the edges of its strips, column tiles and channel
counts, against the FP64 convolution."""
import numpy as np
import pytest
import torch

from deepcharacters_b200.losses import smooth_image
from test_losses_gpu import smooth_fp64  # same directory

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [1, 2, 3, 4, 7, 8, 15])
@pytest.mark.parametrize("n,h,w,c", [(1, 1, 1, 3), (1, 64, 171, 3), (2, 65, 129, 4), (1, 9, 520, 1), (1, 130, 43, 2)])
def test_smooth_matches_fp64_at_tile_edges(size, n, h, w, c):
    img = np.random.default_rng(size).uniform(0, 1, size=(n, h, w, c)).astype(np.float32)
    ours = smooth_image(torch.from_numpy(img).to("cuda:0"), size, 0.2, 0.5 * size).cpu().numpy()
    # values in [0, 1], two FP32 sums of at most 31 terms
    assert np.abs(ours - smooth_fp64(img, size, 0.2, 0.5 * size)).max() < 2e-6
