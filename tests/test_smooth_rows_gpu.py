"""Smoothing of rows with more floats than 32 bits count: the same values as a part of
the row alone, also where the columns of one launch end and at both ends of the row."""
import pytest
import torch

from deepcharacters_b200.losses import smooth_image

pytestmark = pytest.mark.gpu


def test_row_beyond_two_to_the_31_floats():
    s, W = 3, (1 << 31) // 3 + 1000
    g = torch.Generator("cuda:0").manual_seed(5)
    x = torch.rand((1, 1, W, 3), device="cuda:0", generator=g)
    got = smooth_image(x, s, 0.0, 1.5)
    for c in (0, (1 << 30) // 3, (1 << 31) // 3, W):
        lo, hi = max(c - 400, 0), min(c + 400, W)
        a, b = max(lo - s, 0), min(hi + s, W)
        want = smooth_image(x[:, :, a:b].contiguous(), s, 0.0, 1.5)[:, :, lo - a:hi - a]
        assert torch.equal(got[:, :, lo:hi], want)
