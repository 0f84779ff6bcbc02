"""The gradient from signs in groups of 128 pixels a warp: sizes around one and
several groups, against the pair without scratch."""
import numpy as np
import pytest
import torch

from deepcharacters_b200 import _lib
from deepcharacters_b200.losses import image_l1_loss

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("n", [126, 127, 128, 129, 255, 256, 8 * 128 + 1, 300_000, 148 * 8 * 8 * 128 * 2 + 131])
def test_gradient_equals_the_pair_without_scratch(n):
    g = torch.Generator(device=DEV).manual_seed(n)
    r, t = (torch.rand((n, 3), device=DEV, generator=g) for _ in range(2))
    t[::5] = r[::5]
    face = torch.randint(-1, 3, (n,), device=DEV, generator=g, dtype=torch.int32)
    loss, grad = image_l1_loss(r, t, face, None)
    ws, l2, g2 = torch.empty(2, device=DEV, dtype=torch.float64), torch.empty(1, device=DEV), torch.empty_like(grad)
    _lib.call("hc_image_l1_loss", torch.cuda.current_stream().cuda_stream, n, r.data_ptr(), t.data_ptr(),
              face.data_ptr(), None, ws.data_ptr(), l2.data_ptr(), g2.data_ptr())
    assert torch.equal(grad, g2)
    assert abs(float(l2) - float(loss)) <= 1e-6 * max(float(l2), 1.0)
    assert np.isfinite(float(loss)) and int(torch.count_nonzero(grad)) > 0
