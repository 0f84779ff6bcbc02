"""Handles give back all of their device memory."""
import numpy as np
import pytest
import torch

from deepcharacters_b200.skinning import Character, SkinningEngine

pytestmark = pytest.mark.gpu


def test_skinning_handles_give_back_their_memory():
    n, s, k = 200_000, 9, 4
    rng = np.random.default_rng(0)
    v = rng.normal(0, 100, (n, 3)).astype(np.float32)
    ch = Character(np.arange(-1, s - 1, dtype=np.int32), np.zeros(s, np.int32), np.ones((s, 3)),
                   np.tile([[0, 0, 1.0]], (s, 1)), np.arange(s + 1), np.arange(s), np.ones(s), np.arange(s), v, v / 100,
                   rng.integers(0, s, (n, k)))
    SkinningEngine(ch)  # made and dropped
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    for _ in range(20):
        SkinningEngine(ch)
    torch.cuda.synchronize()
    assert before - torch.cuda.mem_get_info()[0] < 32 << 20  # 6.4 MB of base vertices and normals in each
