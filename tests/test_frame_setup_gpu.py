"""The launches that prepare a call: ranges filled by spare blocks at any
alignment and size, and the UV maps from normals normalised once per vertex
against normalising them at every texel."""
import numpy as np
import pytest
import torch

from deepcharacters_b200 import synthetic as S
from deepcharacters_b200.renderer import RendererEngine

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TEX = 37


def _args(sc, B):
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)  # noqa: E731
    return t(sc["verts"]), t(sc["colors"]), torch.zeros((B, TEX, TEX, 3), device=DEV), t(sc["sh"]), t(sc["extr"]), t(
        sc["intr"])


def _engine(sc, mode, views, w, h):
    return RendererEngine(sc["faces"], sc["texcoords"], sc["N"], views, w, h, "vertexColor", "shadeless", 2, 2, mode)


# outputs at offsets of 0 to 3 words inside a larger buffer, whose other words
# have to stay: head, body and tail of a fill, and fills of less than a vector
@pytest.mark.parametrize("w,h,offset", [(1, 1, 0), (1, 1, 3), (3, 1, 1), (7, 5, 2), (96, 80, 0), (97, 83, 1),
                                        (257, 129, 3)])
def test_fills_cover_their_ranges_only(w, h, offset):
    sc = S.render_scene(2, batch=1, views=1, width=w, height=h, seed=5, texture_size=TEX)
    eng = _engine(sc, "face", 1, w, h)
    big = {k: torch.full((w * h * c + 8,), 7, device=DEV, dtype=d)
           for k, c, d in (("bary", 2, torch.float32), ("face", 1, torch.int32), ("render", 3, torch.float32))}
    img = eng.image_shape(1)
    out = {k: big[k][offset:offset + w * h * c].view(img + ((c,) if c > 1 else ()))
           for k, c in (("bary", 2), ("face", 1), ("render", 3))}
    eng.forward(*_args(sc, 1), out=out)
    torch.cuda.synchronize()
    for k, c, want in (("bary", 2, 0), ("face", 1, -1), ("render", 3, 0)):
        n = w * h * c
        assert bool((big[k][offset:offset + n] == want).all()), k
        assert bool((big[k][:offset] == 7).all()) and bool((big[k][offset + n:] == 7).all()), k


# a capture does not allocate: at more frames than the engine has room for it
# takes the normals as they are and normalises at the texel; the same values
@pytest.mark.parametrize("frames", [1, 3, 4, 5, 9])
@pytest.mark.parametrize("views", [1, 2])
def test_uv_normals_once_per_vertex(frames, views):
    B = frames + 1
    sc = S.render_scene(3, batch=B, views=views, width=40, height=32, seed=21, texture_size=TEX)
    args = _args(sc, B)
    eng = _engine(sc, "normal", views, 40, 32)
    want = eng.forward(*args)
    small = _engine(sc, "normal", views, 40, 32)
    small.forward(*(a[:1].contiguous() for a in args))  # texel table and room for one frame
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        got = small.forward(*args)
    g.replay()
    torch.cuda.synchronize()
    assert float(want[4].abs().sum()) > 0
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    del g
