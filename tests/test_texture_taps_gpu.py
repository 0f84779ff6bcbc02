"""Texture-gradient taps of the adjoint where the whole part of (y + j) w + (x + i)
depends on its rounding: the position gradient follows the stated one (the product
rounded first with shading, the sum alone without), against the closed form in FP64
over the same texels.  One pixel and one triangle per frame; random texels, so a tap
beside the stated one changes the gradient as a whole."""
import numpy as np
import pytest
import torch

from deepcharacters_b200.renderer import RendererEngine, renderer_backward

pytestmark = pytest.mark.gpu
DEV, TW, TH, f32 = "cuda:0", 1000, 100, np.float32
TC = np.array([0.03, 0.05, 0.95, 0.12, 0.3, 0.9], f32)
UV = np.stack([TC[0::2], f32(1) - TC[1::2]], 1)  # per corner


def _fma(a, b, c):  # the product of two floats is exact in a long double
    return (np.longdouble(a) * np.longdouble(b) + np.longdouble(c)).astype(f32)


def _texel_positions(bary, first):
    a, b = bary.T
    c = f32(1) - a - b
    s = [_fma(t[0], a, t[1] * b) if first else _fma(t[1], b, t[0] * a) for t in UV.T]
    return _fma(UV[2, 0], c, s[0]) * f32(TW), _fma(UV[2, 1], c, s[1]) * f32(TH)


def _taps(x, y, fs, apart):
    k = np.arange(-fs, fs + 1).astype(f32)
    row, col = (y[:, None] + k)[:, :, None], (x[:, None] + k)[:, None, :]
    return (row * f32(TW) + col if apart else _fma(row, f32(TW), col)).astype(np.int64)


def _position_gradient(idx, tex, G, bary, V, d, fs):
    k = np.arange(-fs, fs + 1.0)
    den = k[:, None] ** 2 + k ** 2
    wu = np.divide(k[None, :].repeat(2 * fs + 1, 0), den, out=np.zeros_like(den), where=den > 0)
    I = np.einsum("nyxc,nc->nyx", tex[np.arange(len(idx))[:, None, None], idx], G)
    gu, gv = (np.einsum("nyx,yx->n", I, w) / np.abs(wu).sum() for w in (wu, wu.T))
    gbc = gu[:, None] * UV[:, 0] * TW + gv[:, None] * UV[:, 1] * TH
    v0, v1, v2 = V.transpose(1, 0, 2)
    dn = (d * np.cross(v1 - v0, v2 - v0)).sum(1, keepdims=True)
    r = (gbc[:, :1] - gbc[:, 2:]) * np.cross(d, v1 - v2) / dn + (gbc[:, 1:2] - gbc[:, 2:]) * np.cross(v0 - v2, d) / dn
    weights = np.concatenate([bary, 1 - bary.sum(1, keepdims=True)], 1)
    return weights[:, :, None] * r[:, None]


@pytest.mark.parametrize("shading", ["shadeless", "shaded"])
@pytest.mark.parametrize("fs", [1, 2, 3])
def test_taps_beside_a_texel_border(shading, fs):
    n, rng = 400, np.random.default_rng(fs)
    P = np.array([[-40.0, -60], [90, 2], [-10, 70]]) + rng.uniform(-5, 5, (n, 3, 2))
    # move the triangle until (y w + x) of pixel (0, 0) is near a whole number
    M = np.concatenate([P, np.ones((n, 3, 1))], 2)
    q = np.linalg.solve(M, (UV.astype(np.float64) @ [TW, TH * TW])[None, :, None].repeat(n, 0))[:, :, 0]
    at = q[:, 0] * 0.5 + q[:, 1] * 0.5 + q[:, 2]
    P[:, :, 0] += ((at - np.round(at) + rng.normal(0, 0.004, n)) / q[:, 0])[:, None]
    V = np.concatenate([(P - 4) / 50 * 1500, np.full((n, 3, 1), 1500.0)], 2).astype(f32)
    eng = RendererEngine(np.array([0, 1, 2], np.int32), TC, 3, 1, 8, 8, "textured", shading, 1, fs)
    eng.set_gradient_parity(False)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)  # noqa: E731
    ex = torch.eye(4, device=DEV)[:3].expand(n, 1, 3, 4).contiguous()
    it = torch.tensor([[50.0, 0, 4], [0, 50, 4], [0, 0, 1]], device=DEV).expand(n, 1, 3, 3).contiguous()
    tex = rng.random((n, TH, TW, 3), f32)
    sh = torch.zeros((n, 1, 27), device=DEV)
    sh[..., ::9] = 1  # light of 1 from everywhere
    col, tgt = torch.zeros((n, 3, 3), device=DEV), torch.zeros((n, 1, 8, 8, 3), device=DEV)
    o = eng.forward(t(V), col, t(tex), sh, ex, it)
    g = np.zeros((n, 1, 8, 8, 3), f32)
    g[:, 0, 0, 0] = rng.normal(size=(n, 3))
    got = renderer_backward(eng, t(g), t(V), col, t(tex), sh, tgt, o[3], o[0], o[1], ex, it)[0].double().cpu().numpy()
    assert int((o[1][:, 0, 0, 0] != 0).sum()) == 0
    bary = o[0][:, 0, 0, 0].cpu().numpy()
    idx = {(a, first): _taps(*_texel_positions(bary, first), fs, a) for a in (True, False) for first in (True, False)}
    apart = shading == "shaded"
    sure = (idx[apart, True] == idx[apart, False]).all((1, 2))  # whichever way the texel position is rounded
    differ = sure & (idx[apart, True] != idx[not apart, True]).any((1, 2))
    assert sure.mean() > 0.5 and differ.sum() >= 5
    d = np.tile(np.array([(0.5 - 4) / 50, (0.5 - 4) / 50, 1.0]), (n, 1))
    want = _position_gradient(idx[apart, True], tex.reshape(n, -1, 3).astype(np.float64), g[:, 0, 0, 0].astype(np.float64),
                              bary.astype(np.float64), V.astype(np.float64), d, fs)
    e = np.abs(got - want).max((1, 2))[sure] / np.abs(want).max()
    assert e.max() < 1e-4  # FP32 sums of (2 fs + 1)^2 terms of both signs
