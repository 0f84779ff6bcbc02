"""Level-wise kinematics and the block-wise skinning adjoint: vertex counts at
the block edges, slots per vertex with and without vector staging, joints
with several dofs or none and prismatic joints, against the FP64 oracle, FP64
autograd and the golden reference outputs."""
import dataclasses
import os

import numpy as np
import pytest
import torch

from deepcharacters_b200.skinning import Character, SkinningEngine
from oracle import skinning_oracle as K

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
GOLDEN = os.path.join(os.path.dirname(__file__), "golden", "dq_skinning.npz")


def _t(a):
    return torch.from_numpy(np.ascontiguousarray(a, np.float32)).to(DEV)


def nrel(a, b):
    a, b = (torch.as_tensor(x).double().cpu() for x in (a, b))
    return float((a - b).norm() / max(b.norm().item(), 1e-30))


def _character(n, k, rng):
    J, S = 23, 9
    parent = np.array([-1] + [int(rng.integers(max(0, j - 4), j)) for j in range(1, J)], np.int32)
    kind = (rng.random(J) < 0.25).astype(np.int32)  # some prismatic
    axis = rng.normal(size=(J, 3))
    axis /= np.linalg.norm(axis, axis=1, keepdims=True)
    # 17 dofs, some driving several joints; some joints driven by several dofs, some by none
    sizes = rng.integers(1, 4, size=17)
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
    dj = rng.integers(0, J - 2, size=off[-1]).astype(np.int32)
    v = rng.normal(0, 500.0, size=(n, 3))
    nr = v / np.linalg.norm(v, axis=1, keepdims=True)
    idx = np.stack([rng.permutation(S)[:k] for _ in range(n)]).astype(np.int32)
    idx[idx == 4] = 5  # a bone without vertices, and repeated slots
    return Character(parent, kind, rng.normal(0, 100.0, size=(J, 3)).astype(np.float32), axis.astype(np.float32), off,
                     dj, rng.uniform(0.5, 1.5, off[-1]).astype(np.float32),
                     rng.permutation(J)[:S].astype(np.int32), v.astype(np.float32), nr.astype(np.float32), idx)


def _autograd_weights(ch, dq, w, g):
    """d (sum v . g) / d weights of the sign-aligned normalised blend, FP64."""
    q = torch.from_numpy(dq)[:, torch.from_numpy(ch.skin_index).long()]
    w = torch.from_numpy(w).double().requires_grad_()
    sign = torch.where((q[..., :1, :4] * q[..., :4]).sum(-1, keepdim=True) < 0, -1.0, 1.0)
    b = (w[..., None] * q * sign).sum(-2)
    b = b / b[..., :4].norm(dim=-1, keepdim=True)
    r, t, p = b[..., :4], b[..., 4:], torch.from_numpy(ch.base_vertices).double()
    u, s = r[..., :3], r[..., 3:]
    rot = p + 2 * torch.linalg.cross(u, torch.linalg.cross(u, p.expand_as(u)) + s * p)
    tr = 2 * (s * t[..., :3] - t[..., 3:] * u + torch.linalg.cross(u, t[..., :3]))
    return torch.autograd.grad(((rot + tr) * torch.from_numpy(g).double()).sum(), w)[0]


def _dof_gradient(ch, v, g, w, gpos, gaxis):
    """Sum over a dof's entries (a joint may be listed twice) of the oracle's gradient of that joint alone."""
    J = ch.n_joints
    one = dataclasses.replace(ch, dof_offsets=np.arange(J + 1, dtype=np.int32), dof_joint=np.arange(J, dtype=np.int32),
                              dof_weight=np.ones(J, np.float32))
    gj = K.dof_grad_reference(one, v, g, w, gpos, gaxis)
    return np.stack([gj[:, ch.dof_joint[a:z]].sum(1) for a, z in zip(ch.dof_offsets, ch.dof_offsets[1:])], 1)


@pytest.mark.parametrize("n,k", [(1, 4), (255, 4), (256, 4), (257, 3), (700, 1), (513, 6)])
def test_kinematics_and_adjoints_match_the_oracle(n, k):
    rng = np.random.default_rng(100 * n + k)
    ch = _character(n, k, rng)
    B = 3
    dofs = rng.uniform(-0.6, 0.6, size=(B, 17)).astype(np.float32)
    w = rng.dirichlet(np.ones(k), size=(B, n)).astype(np.float32)
    g = rng.normal(size=(B, n, 3)).astype(np.float32)
    disp = rng.normal(size=(B, n, 3)).astype(np.float32)
    eng = SkinningEngine(ch, parity=False)
    v, _, gp, ga, dq, _ = eng.dq_forward(_t(dofs), _t(w))
    _, _, gpos, gaxis = K.fk(ch, dofs)
    dq_o = K.dual_quaternions(ch, dofs)
    assert nrel(gp, gpos) < 1e-5 and nrel(ga, gaxis) < 1e-5
    # a quaternion and its negative are the same rotation
    flip = np.sign((dq.cpu().numpy()[..., :4] * dq_o[..., :4]).sum(-1, keepdims=True))
    assert nrel(dq * _t(flip), dq_o) < 1e-5
    gd, gw = eng.dq_backward(_t(g), v, gp, ga, dq, _t(w))
    assert nrel(gd, _dof_gradient(ch, v.cpu().numpy(), g, w, gpos, gaxis)) < 1e-5
    if k > 1:
        assert nrel(gw, _autograd_weights(ch, dq.double().cpu().numpy(), w, g)) < 1e-5
    else:  # the normalised blend of one joint does not depend on its weight: zero but for rounding of |v| |g| terms
        assert float((gw[..., 0].abs() / (v.norm(dim=-1) * _t(g).norm(dim=-1))).max()) < 1e-5
    vl, _, gpl, gal, xf, _ = eng.lbs_forward(_t(dofs), _t(w), _t(disp))
    ld, lw, lg = eng.lbs_backward(_t(g), vl, gpl, gal, xf, _t(w), _t(disp))
    assert nrel(ld, _dof_gradient(ch, vl.cpu().numpy(), g, w, gpos, gaxis)) < 1e-5
    Rs, ts = K.skin_transforms(ch, dofs)
    R, t = Rs[:, ch.skin_index], ts[:, ch.skin_index]
    p = ch.base_vertices.astype(np.float64) + disp
    assert nrel(lw, np.einsum("bvki,bvi->bvk", np.einsum("bvkij,bvj->bvki", R, p) + t, g)) < 1e-5
    assert nrel(lg, np.einsum("bvk,bvkji,bvj->bvi", w.astype(np.float64), R, g)) < 1e-5


def test_parity_gradients_match_the_golden_reference_outputs():
    z = np.load(GOLDEN)
    D = z["dofs"].shape[1]
    ch = Character(z["parent"], np.zeros(len(z["parent"]), np.int32), z["offset"], z["axis"],
                   np.arange(D + 1, dtype=np.int32), z["dof_joint"], z["dof_weight"], z["skin_joint"], z["verts"],
                   np.tile(np.float32([0, 0, 1]), (len(z["verts"]), 1)), z["skin_index"])
    eng = SkinningEngine(ch)
    gd, gw = eng.dq_backward(_t(z["grad"]), _t(z["out_vertices"]), _t(z["gpos"]), _t(z["gaxis"]), _t(z["dq"]),
                             _t(z["weights"]))
    assert nrel(gd, z["grad_dofs"]) < 1e-5 and nrel(gw, z["grad_weights"]) < 1e-5
