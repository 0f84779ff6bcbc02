"""Pixel rays by their stated order of roundings, read back from barycentrics: the
camera matrix's inverse, the triangle's plane and the weight of its first vertex
(a quarter of the hit's x) scale by powers of two, so nothing but the ray rounds.
The skew makes the two products of the ray's x row round differently by order."""
import numpy as np
import pytest
import torch

from deepcharacters_b200.renderer import RendererEngine

pytestmark = pytest.mark.gpu
DEV, RES, f32 = "cuda:0", 16, np.float32


def _fma(a, b, c):  # the product of two floats is exact in a long double
    return (np.longdouble(a) * np.longdouble(b) + np.longdouble(c)).astype(f32)


def _weight(skew, first):
    u = ((np.arange(RES) + 0.5) * 1000).astype(f32)[None, None, :]
    v = u.transpose(0, 2, 1)
    m0, m1 = f32(1 / 64), (-skew / f32(4096))[:, None, None]
    x = _fma(m1, v, m0 * u) if first else _fma(m0, u, m1 * v)
    y = np.broadcast_to(v * m0, x.shape)
    length2 = _fma(f32(1000), f32(1000), _fma(x, x, y * y))
    r = torch.rsqrt(torch.from_numpy(length2).to(DEV)).cpu().numpy()
    return f32(0.25) * ((f32(2) / (f32(1000) * r)) * (x * r))


@pytest.mark.parametrize("tile", [8, 16, 32])
@pytest.mark.parametrize("diagnostics", [False, True])
def test_barycentrics_of_skewed_cameras(tile, diagnostics):
    n = 2000
    skew = -np.random.default_rng(tile).uniform(0.5, 12, n).astype(f32)
    K = np.tile(np.diag([64, 64, 1]).astype(f32), (n, 1, 1, 1))
    K[:, 0, 0, 1] = skew
    eng = RendererEngine(np.array([0, 1, 2], np.int32), None, 3, 1, RES, RES, "vertexColor", "shadeless", 1, 1)
    eng.set_tuning(tile, 64)
    verts = torch.tensor([[4000.0, 0, 2000], [0, -4000, 2000], [0, 4000, 2000]], device=DEV).expand(n, 3, 3).contiguous()
    extr = torch.eye(4, device=DEV)[:3].expand(n, 1, 3, 4).contiguous()
    out = eng.forward(verts, torch.rand((n, 3, 3), device=DEV), None, None, extr, torch.from_numpy(K).to(DEV),
                      diagnostics=diagnostics)
    assert int((out[1] != 0).sum()) == 0
    got, want, other = out[0][:, 0, :, :, 0].cpu().numpy(), _weight(skew, True), _weight(skew, False)
    assert np.array_equal(got, want)
    assert (want != other).mean() > 0.01  # the order matters
