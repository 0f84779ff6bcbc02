"""UV maps of several texture sizes on one engine, captured and eager: every call
and every replay gives the maps of its own size."""
import numpy as np
import pytest
import torch

from deepcharacters_b200 import synthetic as S
from deepcharacters_b200.renderer import RendererEngine

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _scene(mode):
    sc = S.render_scene(3, batch=2, views=1, width=40, height=32, seed=21, texture_size=8)
    t = lambda k: torch.from_numpy(np.ascontiguousarray(sc[k])).to(DEV)  # noqa: E731
    make = lambda: RendererEngine(sc["faces"], sc["texcoords"], sc["N"], 1, 40, 32, "vertexColor", "shadeless",  # noqa: E731
                                  2, 2, mode)
    x = [t(k) for k in ("verts", "colors", "sh", "extr", "intr")]

    def run(eng, size):
        return eng.forward(x[0], x[1], torch.zeros((2, size, size, 3), device=DEV), *x[2:])[4]

    return make, run, lambda size: run(make(), size)


def _graph(f):
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = f()
    return g, out


def _replayed(g, out):
    out.zero_()
    g.replay()
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("mode", ["normal", "face"])
@pytest.mark.parametrize("other", [16, 64])
def test_replay_after_another_size(mode, other):
    make, run, fresh = _scene(mode)
    eng, want = make(), fresh(37)
    run(eng, 37)
    g, out = _graph(lambda: run(eng, 37))
    assert torch.equal(run(eng, other), fresh(other))
    assert torch.equal(_replayed(g, out), want)
    assert torch.equal(run(eng, 37), want) and torch.equal(run(eng, other), fresh(other))


def test_size_first_seen_by_a_capture():
    make, run, fresh = _scene("normal")
    eng = make()
    run(eng, 64)
    g, out = _graph(lambda: run(eng, 37))  # the 64^2 table has the room; the graph builds the 37^2 one
    assert torch.equal(run(eng, 37), fresh(37)) and torch.equal(run(eng, 64), fresh(64))
    g2, out2 = _graph(lambda: run(eng, 20))
    for _ in range(2):
        assert torch.equal(_replayed(g, out), fresh(37)) and torch.equal(_replayed(g2, out2), fresh(20))
        assert torch.equal(run(eng, 64), fresh(64))
