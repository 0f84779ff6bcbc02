"""The image L1 with per-pixel scratch: remainders, masks, unaligned views, no
valid pixel, and the pair without scratch, against FP64."""
import numpy as np
import pytest
import torch

from deepcharacters_b200 import _lib
from deepcharacters_b200.losses import image_l1_loss

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("offset", [0, 1])  # pixels: 1 leaves no buffer 16-byte aligned
@pytest.mark.parametrize("n,masked", [(1, False), (3, True), (4, False), (5, True), (1027, True), (40_001, False)])
def test_l1_matches_fp64(n, masked, offset):
    rng = np.random.default_rng(n)
    r, t = (torch.from_numpy(rng.uniform(0, 1, size=(n + offset, 3)).astype(np.float32)).to(DEV)[offset:]
            for _ in range(2))
    t[::5] = r[::5]  # exact zeros are not counted
    face = torch.from_numpy(rng.integers(-1, 3, size=n + offset).astype(np.int32)).to(DEV)[offset:]
    mask = torch.from_numpy(rng.integers(0, 2, size=n).astype(np.uint8)).to(DEV) if masked else None
    loss, grad = image_l1_loss(r, t, face, mask)
    on = ((face >= 0) & (mask != 0 if masked else True))[:, None]
    # each product rounded on its own, as the op does
    d = ((r * 255.0).double() - (t * 255.0).double()) * on
    count = int(torch.count_nonzero(d))
    want = float(d.abs().sum()) / count if count else 0.0
    assert abs(float(loss) - want) <= 1e-6 * max(want, 1.0)  # FP32 sums per thread, FP64 beyond
    scale = np.float32(255.0) / np.float32(count) if count else np.float32(0)
    assert torch.equal(grad, d.sign().float() * float(scale))
    ws, l2, g2 = torch.empty(2, device=DEV, dtype=torch.float64), torch.empty(1, device=DEV), torch.empty_like(grad)
    _lib.call("hc_image_l1_loss", torch.cuda.current_stream().cuda_stream, n, r.data_ptr(), t.data_ptr(),
              face.data_ptr(), _lib.ptr(mask), ws.data_ptr(), l2.data_ptr(), g2.data_ptr())
    assert torch.equal(grad, g2) and abs(float(l2) - float(loss)) <= 1e-6 * max(want, 1.0)


def test_l1_without_a_valid_pixel():
    r, t = torch.rand((9, 3), device=DEV), torch.rand((9, 3), device=DEV)
    loss, grad = image_l1_loss(r, t, torch.full((9,), -1, device=DEV, dtype=torch.int32))
    assert float(loss) == 0.0 and float(grad.abs().max()) == 0.0
    with pytest.raises(_lib.HcError):  # empty tensors have no address
        image_l1_loss(r[:0], t[:0], torch.empty(0, device=DEV, dtype=torch.int32))
