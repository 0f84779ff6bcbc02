"""Coverage of pixels whose barycentric is the tolerance (-0.001) to the last bits: the
boundary op decides them by a stated order of roundings, the same in a tile's bin and
in the sweep of a small box beyond it, and with the products apart in the sweep of a
box of more than nine tiles.  One triangle and one vertex per frame, at the test
pixel; eight more triangles cover the pixels around it."""
import numpy as np
import pytest
import torch

from deepcharacters_b200.silhouette import MeshBoundaryEngine

pytestmark = pytest.mark.gpu
DEV, RES, f32 = "cuda:0", 64, np.float32


def _fma(a, b, c):  # the product of two floats is exact in a long double
    return (a.astype(np.longdouble) * b.astype(np.longdouble) + c.astype(np.longdouble)).astype(f32)


def _covered(V, c, apart):
    a, b, q = V[:, 0], V[:, 1], V[:, 2]

    def numerator(e):
        s = _fma(e[:, 0] - a[:, 0], c[:, 1], (a[:, 1] - e[:, 1]) * c[:, 0])
        if apart:
            return (s + a[:, 0] * e[:, 1]) - e[:, 0] * a[:, 1]
        return _fma(-e[:, 0], a[:, 1], _fma(a[:, 0], e[:, 1], s))

    def denominator(e, o, first):
        x, y, u, v = a[:, 1] - e[:, 1], e[:, 0] - a[:, 0], o[:, 0], o[:, 1]
        s = _fma(x, u, y * v) if first else _fma(y, v, x * u)
        return _fma(-e[:, 0], a[:, 1], _fma(a[:, 0], e[:, 1], s))

    e2 = numerator(b) / denominator(b, q, True)
    e1 = numerator(q) / denominator(q, b, False)
    e0 = f32(1) - e2 - e1
    return np.logical_and.reduce([(e >= f32(-0.001)) & (e <= f32(1.001)) for e in (e0, e1, e2)])


def _triangles(rng, n, small):
    """Test pixels in a corner of their tile, and triangles with one weight of about -0.001 there."""
    T = 8 * rng.integers(3, 5, (n, 2)) + rng.integers(1, 3, (n, 2))
    c, s = T + 0.5, 9 if small else 60
    a, b, k = c + rng.uniform(-s, s, (n, 2)), c + rng.uniform(-s, s, (n, 2)), rng.integers(0, 3, n)
    w, e, i = rng.dirichlet([1, 1], n), -0.001 + rng.normal(0, 1e-6 if small else 3e-6, n), np.arange(n)
    o, p = (k + 1) % 3, (k + 2) % 3
    V = np.empty((n, 3, 2))
    V[i, k], V[i, o] = a, b
    V[i, p] = (c - e[:, None] * a - ((1 - e) * w[:, 0])[:, None] * b) / ((1 - e) * w[:, 1])[:, None]
    V = V.astype(f32)
    lo, hi = V.min(1), V.max(1)
    tiles = np.prod(np.minimum(hi + 0.5, RES - 1).astype(int) // 8 - np.maximum(lo - 0.5, 0).astype(int) // 8 + 1, 1)
    ok = (np.abs(V).max((1, 2)) < 200) & (w.min(1) > 0.06) & (lo - 0.5 <= T).all(1) & (hi + 0.5 >= T + 1).all(1)
    ok &= (tiles > 1) & (tiles <= 9) if small else tiles > 16
    return T[ok][:1200], V[ok][:1200]


@pytest.mark.parametrize("small", [True, False])
@pytest.mark.parametrize("swept", [False, True])
def test_pixels_at_the_tolerance(small, swept):
    T, V = _triangles(np.random.default_rng(8), 40_000, small)
    n, more = len(T), 2500 if swept else 0  # triangles that fill the tile's bin first
    pts = np.full((n, 28 + 3 * more, 2), -1000.0, f32)
    around = [(x, y) for y in (-1, 0, 1) for x in (-1, 0, 1) if (x, y) != (0, 0)]
    for k, d in enumerate(around):
        pts[:, 3 * k:3 * k + 3] = (T + 0.5 + d)[:, None] + np.array([[-0.3, -0.25], [0.3, -0.25], [0, 0.35]])
    pts[:, 24:27], pts[:, 27] = V, T + 0.5
    inside = np.random.default_rng(0).uniform(0, 0.6, (3 * more, 2)) + 6.2  # of the tile, away from the pixels
    pts[:, 28:] = (T // 8 * 8)[:, None] + inside
    faces = np.concatenate([np.arange(28, 28 + 3 * more), np.arange(27)]).reshape(-1, 3)
    eng = MeshBoundaryEngine(faces, pts.shape[1])
    p = torch.from_numpy(pts).to(DEV).reshape(n, 1, -1, 2)
    extr = torch.eye(4, device=DEV)[:3].expand(n, 1, 3, 4).contiguous()
    intr = torch.eye(3, device=DEV).expand(n, 1, 3, 3).contiguous()
    flags = eng.forward(torch.zeros((n, pts.shape[1], 3), device=DEV), extr, intr, RES, RES, points_image_space=p)
    got, c = flags[:, 0, 27].cpu().numpy() == 0, (T + 0.5).astype(f32)
    want, other = (_covered(V, c, apart) for apart in (swept and not small, not (swept and not small)))
    assert np.array_equal(got, want)
    assert 0.3 < want.mean() < 0.7 and (want != other).sum() >= 5  # both roundings occur
