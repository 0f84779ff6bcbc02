"""Joint angle gradients where frames times dofs pass 2^27: a warp each, more than
2^32 threads."""
import numpy as np
import pytest
import torch

from deepcharacters_b200.skinning import Character, SkinningEngine

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("node_level", [False, True])
def test_gradients_of_many_frames_and_dofs(node_level):
    B, s, n, D = 65535, 2, 3, 2100
    rng = np.random.default_rng(3)
    v = rng.normal(0, 100, (n, 3)).astype(np.float32)
    off = np.zeros(D + 1, np.int32)
    off[1:], off[-1] = 1, 2  # the first dof drives joint 0, the last one joint 1, the others none
    eng = SkinningEngine(Character(np.array([-1, 0], np.int32), np.zeros(s, np.int32), np.ones((s, 3)),
                                   np.tile([[0, 0, 1.0]], (s, 1)), off, np.arange(s), np.ones(s), np.arange(s), v,
                                   v / 100, np.tile([[0, 1]], (n, 1))))
    g = torch.Generator(DEV).manual_seed(4)
    w = torch.full((n, s), 0.5, device=DEV)
    gv = torch.randn((B, n, 3), device=DEV, generator=g)

    def grad(lo, hi):
        dofs = torch.zeros((hi - lo, D), device=DEV)
        if node_level:
            nodes = torch.arange(n, dtype=torch.int32, device=DEV)
            return eng.pose2eg_backward(dofs, nodes, w, gv[lo:hi].contiguous(), gv[lo:hi].contiguous())
        ws = w.expand(hi - lo, n, s).contiguous()
        o = eng.dq_forward(dofs, ws)
        return eng.dq_backward(gv[lo:hi].contiguous(), o[0], o[2], o[3], o[4], ws)[0]

    got = grad(0, B)
    for lo, hi in ((0, 2000), (63800, B)):  # the values in FP32 sums of another order
        want = grad(lo, hi)
        assert float((got[lo:hi] - want).abs().max()) <= 1e-5 * float(want.abs().max())
        assert float(want[:, -1].abs().min()) > 0 and float(want[:, 1:-1].abs().max()) == 0
