"""The embedded graph's fused vertex pass and moment-based node pass: vertex
counts at the block edge, vertices without nodes, ragged lists, nodes without
vertices, with and without markers and skinned gradients, against FP64
autograd."""
import numpy as np
import pytest
import torch

from deepcharacters_b200.embedded_graph import EGData, EmbeddedGraphEngine

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def nrel(a, b):
    a, b = a.double().cpu(), b.double().cpu()
    return float((a - b).norm() / max(b.norm().item(), 1e-30))


def _euler(a):
    c, s, one, zero = a.cos(), a.sin(), torch.ones_like(a[..., 0]), torch.zeros_like(a[..., 0])
    m = lambda *e: torch.stack(e, -1).reshape(*one.shape, 3, 3)  # noqa: E731
    x = m(one, zero, zero, zero, c[..., 0], -s[..., 0], zero, s[..., 0], c[..., 0])
    y = m(c[..., 1], zero, s[..., 1], zero, one, zero, -s[..., 1], zero, c[..., 1])
    z = m(c[..., 2], -s[..., 2], zero, s[..., 2], c[..., 2], zero, zero, zero, one)
    return z @ y @ x


@pytest.mark.parametrize("full", [False, True])
@pytest.mark.parametrize("n,m,markers", [(5, 2, 0), (127, 9, 2), (128, 40, 0), (300, 33, 5)])
def test_adjoint_matches_fp64_autograd(n, m, markers, full):
    rng = np.random.default_rng(n)
    base = rng.normal(0, 500.0, size=(n, 3)).astype(np.float32)
    faces = np.stack([rng.permutation(n)[:3] for _ in range(2 * n)]).astype(np.int32)
    sizes = rng.integers(0, 6, size=n).astype(np.int32)  # some vertices without nodes
    sizes[0] = 3
    off = np.concatenate([[0], np.cumsum(sizes)[:-1]]).astype(np.int32)
    vid = np.repeat(np.arange(n, dtype=np.int32), sizes)
    idx = rng.integers(0, max(m - 1, 1), size=len(vid)).astype(np.int32)  # the last node gets no vertex
    w = rng.uniform(0.1, 1.0, size=len(vid)).astype(np.float32)
    order = np.lexsort((vid, idx))
    nsz = np.bincount(idx, minlength=m).astype(np.int32)
    noff = np.concatenate([[0], np.cumsum(nsz)[:-1]]).astype(np.int32)
    nodes = rng.permutation(n)[:m].astype(np.int32)
    mk = rng.normal(0, 500.0, size=(markers, 3)).astype(np.float32) if markers else None
    mn = rng.permutation(m)[:markers].astype(np.int32) if markers else None
    eng = EmbeddedGraphEngine(EGData(base, faces, nodes, off, sizes, idx, w, noff, nsz, vid[order], w[order], mk, mn),
                              full_skinned_gradient=full)
    B = 2
    f = lambda s, *shape: torch.from_numpy(rng.normal(0, s, size=shape).astype(np.float32)).to(DEV)  # noqa: E731
    x = [f(10.0, B, m, 3), f(0.3, B, m, 3), f(20.0, B, m, 3), f(0.4, B, m, 3), f(1.0, B, n, 3)]
    gv, gm = f(1.0, B, n, 3), f(1.0, B, max(markers, 1), 3)
    v, _, mkout, _, da, sa = eng.forward(*x)
    ours = eng.backward(gv, gm if markers else None, da, sa, x[0], x[4])
    dT, dA, sT, sA, disp = (t.double().requires_grad_() for t in x)
    t64 = lambda a: torch.from_numpy(a).to(DEV).double()  # noqa: E731
    P, g = t64(base), t64(base)[torch.from_numpy(nodes).long()]
    I, V, W = torch.from_numpy(idx).long().to(DEV), torch.from_numpy(vid).long().to(DEV), t64(w)[None, :, None]
    Rd, Rs = _euler(dA), _euler(sA)
    inner = W * ((Rd[:, I] @ (P[V] - g[I])[None, ..., None])[..., 0] + g[I] + dT[:, I])
    vnr = torch.zeros(B, n, 3, device=DEV, dtype=torch.float64).index_add(1, V, inner) + disp
    outer = W * ((Rs[:, I] @ vnr[:, V, :, None])[..., 0] + sT[:, I])
    want = torch.zeros(B, n, 3, device=DEV, dtype=torch.float64).index_add(1, V, outer)
    assert nrel(v, want) < 1e-5
    loss = (want * gv.double()).sum()
    if markers:
        k = torch.from_numpy(mn).long().to(DEV)
        mu = (Rd[:, k] @ (t64(mk) - g[k])[None, ..., None])[..., 0] + g[k] + dT[:, k]
        mout = (Rs[:, k] @ mu[..., None])[..., 0] + sT[:, k]
        assert nrel(mkout, mout) < 1e-5
        loss = loss + (mout * gm.double()).sum()
    ref = torch.autograd.grad(loss, [dT, dA, sT, sA, disp])
    for k, (a, b) in enumerate(zip(ours, ref)):
        if k in (2, 3) and not full:
            assert float(a.abs().max()) == 0.0
        else:
            assert nrel(a, b) < 1e-5, k
