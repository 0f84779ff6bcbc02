"""Performance cases of the deform-and-render framework.

Each case is one pass of work that a training or rendering program has the
framework do, through its public entry points:

  render   ``RendererEngine.forward`` (free-viewpoint rendering) or
           ``CudaRendererGpu`` with its gradients (a training renderer)
  uv       the UV-space normal map of posed frames (``compute_normal_map``)
  deform   node skinning, embedded-graph deformation and both adjoints
  skin     dual-quaternion or linear-blend vertex skinning and its adjoint
  sil      camera projection, mesh boundary, silhouette loss and adjoints
  images   target smoothing and the masked L1 image loss
  chain    a whole captured training step (``DeformRenderChain``)

Meshes are icospheres in millimetres with per-vertex jitter, posed by a random
24-joint tree, as in ``synthetic.py``; cameras stand on a 3 m ring.  A
character (mesh, skeleton, graph, masks) depends on the sizes alone; poses,
colours, textures, targets and upstream gradients come from the seed.
"""
import functools
import math

import numpy as np
import torch

from deepcharacters_b200 import synthetic as S
from deepcharacters_b200.chain import DeformRenderChain, character, eg_data
from deepcharacters_b200.embedded_graph import EmbeddedGraphEngine, EmbeddedGraphGpu
from deepcharacters_b200.losses import image_l1_loss, smooth_image
from deepcharacters_b200.renderer import CudaRendererGpu, RendererEngine
from deepcharacters_b200.silhouette import (CameraProjectionGpu, MeshBoundaryEngine, MultiViewSilhouetteLossGpu,
                                            SilhouetteEngine)
from deepcharacters_b200.skinning import SkinningEngine, dq_skinning_gpu, lb_skinning_gpu

DEV = "cuda"


# ----------------------------------------------------------------------------
# the cases
# ----------------------------------------------------------------------------
def listed():
    return [
        # one view of one frame, forward only: the smallest rendering call (a viewer's frame)
        _case("render_512", "render", subdiv=5, frames=1, views=1, width=512, height=512, albedo="vertexColor",
              shading="shadeless", backward=False, texture=16),
        # a training renderer on a character's static texture, lit by SH: one frame, four cameras
        _case("render_textured_shaded", "render", subdiv=6, frames=1, views=4, width=1024, height=1024,
              albedo="textured", shading="shaded", backward=True, texture=1024),
        # texture optimisation at high resolution: bilinear sampling and its adjoint into the texture
        _case("render_hires_bilinear", "render", subdiv=7, frames=1, views=4, width=2048, height=2048,
              albedo="texturedBilinear", shading="shadeless", backward=True, texture=1024),
        # vertex colours under SH lighting at an odd camera size, a small batch
        _case("render_shaded_odd", "render", subdiv=5, frames=3, views=3, width=643, height=477,
              albedo="vertexColor", shading="shaded", backward=True, texture=16),
        # UV-space normal maps of a few posed frames (the texture network's input)
        _case("uv_normal_map", "uv", subdiv=6, frames=4, texture=512),
        # one frame of a tracked character: pose to embedded graph to vertices and back
        _case("deform_1", "deform", subdiv=5, nodes=300, frames=1),
        # a training batch of the same at the larger character
        _case("deform_16", "deform", subdiv=6, nodes=1000, frames=16),
        # a training batch of vertex skinning, gradients to joint angles and skin weights
        _case("skin_dq_16", "skin", mode="dq", subdiv=6, frames=16),
        # the silhouette term of a small batch, eagerly
        _case("silhouette_4x4", "sil", subdiv=6, frames=4, views=4, width=1024, height=1024),
        # target smoothing and the image loss of one frame's cameras
        _case("images_8", "images", images=8, width=1024, height=1024, size=3),
        # a small mixed-resolution batch of the vertex-skinned character, one captured step
        _case("chain_mixed_2x4", "chain", deformation="dq", subdiv=5, nodes=300, frames=2, views=4, width=0, height=0,
              parity=False),
        # the training batch: 16 frames x 8 cameras at 1024 x 1024, one captured step
        _case("chain_16x8", "chain", deformation="eg", subdiv=6, nodes=1000, frames=16, views=8, width=1024,
              height=1024, parity=True),
    ]


def draw(rng):
    """One more case of the ranges that the listed ones stand for."""
    kind = rng.choice(("render", "render", "render", "uv", "deform", "deform", "skin", "skin", "sil", "images",
                       "chain", "chain"))
    if kind == "render":
        subdiv, texture = rng.randint(4, 7), _log_int(rng, 16, 1024)
        width, height = _log_int(rng, 200, 2048), _log_int(rng, 200, 2048)
        frames, views = _batch(rng, 16, 8, 4 * 2048 * 2048 // (width * height))
        albedo = rng.choice(("vertexColor", "vertexColor", "textured", "texturedBilinear", "normal", "depth"))
        return _case(None, kind, subdiv=subdiv, frames=frames, views=views, width=width, height=height, albedo=albedo,
                     shading=rng.choice(("shaded", "shadeless")), texture=texture,
                     backward=albedo not in ("normal", "depth") and rng.random() < 0.75)
    if kind == "uv":
        return _case(None, kind, subdiv=rng.randint(4, 7), frames=_log_int(rng, 1, 16),
                     texture=_log_int(rng, 100, 1024))
    if kind == "deform":
        return _case(None, kind, subdiv=rng.randint(4, 6), nodes=_log_int(rng, 60, 1000), frames=_log_int(rng, 1, 32))
    if kind == "skin":
        return _case(None, kind, mode=rng.choice(("dq", "lbs")), subdiv=rng.randint(4, 7),
                     frames=_log_int(rng, 1, 32))
    if kind == "images":
        return _case(None, kind, images=_log_int(rng, 1, 32), width=_log_int(rng, 100, 1536),
                     height=_log_int(rng, 100, 1024), size=rng.randint(1, 7))
    width, height = _log_int(rng, 200, 1536), _log_int(rng, 200, 1024)
    mixed = kind == "chain" and rng.random() < 0.3
    pixels = 1024 * 1024 if mixed else width * height
    frames, views = _batch(rng, 16, 8, 64 * 1024 * 1024 // pixels)
    subdiv = rng.randint(4, 6)
    if kind == "sil":
        return _case(None, kind, subdiv=subdiv, frames=frames, views=views, width=width, height=height)
    return _case(None, kind, deformation=rng.choice(("eg", "dq")), subdiv=subdiv, nodes=_log_int(rng, 60, 1000),
                 frames=frames, views=views, width=0 if mixed else width, height=0 if mixed else height,
                 parity=rng.random() < 0.5)


def _case(name, kind, **k):
    c = dict(kind=kind, **k)
    if name:
        c["name"] = name
    return c


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _batch(rng, most_frames, most_views, most):
    """(frames, views) with at most ``most`` views in all."""
    views = _log_int(rng, 1, max(1, min(most_views, most)))
    return _log_int(rng, 1, max(1, min(most_frames, most // views))), views


# ----------------------------------------------------------------------------
# characters (by sizes) and inputs (by seed)
# ----------------------------------------------------------------------------
@functools.lru_cache(maxsize=8)
def _mesh(subdiv):
    v, f = S.icosphere(subdiv)
    return v, f, S.sphere_mesh(subdiv, S.rng_for(2))[0]


@functools.lru_cache(maxsize=8)
def _texcoords(subdiv):
    v, f, _ = _mesh(subdiv)
    return S.spherical_uvs(v.astype(np.float32), f)


@functools.lru_cache(maxsize=8)
def _skeleton(subdiv):
    rng = S.rng_for(2, 7)
    sk = S.random_skeleton(24, rng)
    return (sk,) + S.skinning_weights(_mesh(subdiv)[2], sk, 4, rng)


@functools.lru_cache(maxsize=8)
def _graph(subdiv, nodes):
    """Farthest-point nodes, each vertex on its four nearest with inverse-distance weights."""
    v = torch.from_numpy(_mesh(subdiv)[2]).to(DEV, torch.float64)
    N, M = v.shape[0], min(nodes, v.shape[0] // 4)
    pick = torch.zeros(M, dtype=torch.int64, device=DEV)
    near = torch.full((N,), math.inf, device=DEV, dtype=torch.float64)
    for i in range(1, M):
        near = torch.minimum(near, (v - v[pick[i - 1]]).norm(dim=1))
        pick[i] = near.argmax()
    dist, idx = torch.cat([torch.stack([x.double() for x in torch.cdist(c, v[pick]).topk(4, dim=1, largest=False)])
                           for c in v.split(16384)], dim=1)
    w = 1.0 / dist.clamp_min(1e-3)
    w = (w / w.sum(1, keepdim=True)).cpu().numpy().astype(np.float32).reshape(-1)
    idx = idx.cpu().numpy().astype(np.int32).reshape(-1)
    vid = np.repeat(np.arange(N, dtype=np.int32), 4)
    order = np.lexsort((vid, idx))
    sizes = np.bincount(idx, minlength=M).astype(np.int32)
    offsets = np.concatenate([[0], np.cumsum(sizes)[:-1]]).astype(np.int32)
    return S.EmbeddedGraph(pick.cpu().numpy().astype(np.int32), (np.arange(N) * 4).astype(np.int32),
                           np.full(N, 4, np.int32), idx, w, offsets, sizes, vid[order], w[order])


@functools.lru_cache(maxsize=16)
def _masks(width, height):
    return torch.from_numpy(S.silhouette_masks(1, 3, width, height, seed=2, scale=min(width, height) / 512.0)[0])


def _scene(subdiv, nodes):
    """The character part of ``synthetic.chain_scene``."""
    sk, idx, w = _skeleton(subdiv)
    _, faces, verts = _mesh(subdiv)
    g = _graph(subdiv, nodes)
    mk = np.linspace(0, g.n_nodes - 1, 8).astype(np.int32)
    return dict(verts=verts, faces=faces, graph=g, markers=verts[g.node_vertex[mk]] + np.float32(3.0), marker_node=mk,
                skeleton=sk, skin_index=idx, skin_weights=w)


class _Draws:
    """Device random numbers of one seed."""

    def __init__(self, seed):
        self.g = torch.Generator(DEV).manual_seed(int(seed))

    def normal(self, std, *shape):
        return torch.randn(shape, device=DEV, generator=self.g) * std

    def uniform(self, lo, hi, *shape):
        return torch.rand(shape, device=DEV, generator=self.g) * (hi - lo) + lo

    def image(self, *shape):
        """8-bit image values / 255."""
        return torch.randint(0, 256, shape, device=DEV, generator=self.g, dtype=torch.uint8).float().div_(255.0)

    def masks(self, frames, sizes):
        """Distance images [frames] x per camera, flipped at random: a list of [B, H, W] per camera."""
        out = []
        for c, (w, h) in enumerate(sizes):
            m = _masks(w, h)[c % 3].to(DEV)
            flips = torch.randint(0, 4, (frames,), generator=self.g, device=DEV).tolist()
            out.append(torch.stack([m.flip([d for d in (0, 1) if f >> d & 1]) for f in flips]))
        return out

    def sh(self, frames, views):
        sh = self.normal(0.1, frames, views, 27)
        sh[..., [0, 9, 18]] = 1.0
        return sh


def _cameras(views, sizes, frames):
    ex, it = [], []
    for c, (w, h) in enumerate(sizes):
        e, i = S.camera_ring(views, 3.0 * S.MM, 600.0 * min(w, h) / 512.0, w, h)
        ex.append(e[12 * c:12 * c + 12])
        it.append(i[9 * c:9 * c + 9])
    tile = lambda a: torch.from_numpy(np.tile(np.concatenate(a)[None], (frames, 1))).to(DEV)  # noqa: E731
    return tile(ex), tile(it)


def _sizes(case):
    if case["width"]:
        return [(case["width"], case["height"])] * case["views"]
    return list(zip(*S.mixed_camera_sizes(case["views"], 3)))


def _posed_mesh(case, d):
    v = torch.from_numpy(_mesh(case["subdiv"])[0]).to(DEV, torch.float32) * S.MM
    return v + d.normal(0.01 * S.MM, case["frames"], *v.shape)


# ----------------------------------------------------------------------------
# render
# ----------------------------------------------------------------------------
def _render_inputs(case, seed):
    d, B, C, W, H, t = _Draws(seed), case["frames"], case["views"], case["width"], case["height"], case["texture"]
    verts = _posed_mesh(case, d)
    ex, it = _cameras(C, _sizes(case), B)
    x = dict(verts=verts, colors=d.uniform(0, 1, *verts.shape), texture=d.uniform(0, 1, B, t, t, 3), sh=d.sh(B, C),
             extr=ex, intr=it)
    if case["backward"]:
        x["target"], x["grad"] = d.image(B, C, H, W, 3), d.normal(1.0, B, C, H, W, 3)
    return x


def _prepare_render(case, seed):
    x = _render_inputs(case, seed)
    _, faces, _ = _mesh(case["subdiv"])
    s = dict(case=case, faces=faces, texcoords=_texcoords(case["subdiv"]), **x)
    if case["backward"]:
        for k in ("verts", "colors", "texture", "sh"):
            s[k].requires_grad_()
    else:
        s["engine"] = RendererEngine(faces, s["texcoords"], x["verts"].shape[1], case["views"], case["width"],
                                     case["height"], case["albedo"], case["shading"], 2, 2)
    return s


def _run_render(s):
    c = s["case"]
    if not c["backward"]:
        return s["engine"].forward(s["verts"], s["colors"], s["texture"], s["sh"], s["extr"], s["intr"])[:4]
    r = CudaRendererGpu(s["faces"], s["texcoords"], s["verts"].shape[1], c["views"], c["width"], c["height"],
                        c["albedo"], c["shading"], 2, 2, "none", s["verts"], s["colors"], s["texture"], s["sh"],
                        s["target"], s["extr"], s["intr"])
    render = r.getRenderBufferTF()
    grads = torch.autograd.grad(render, [s["verts"], s["colors"], s["texture"], s["sh"]], s["grad"])
    return [r.getBaryCentricBufferTF(), r.getFaceBufferTF(), render, r.getVertexNormalTF(), *grads]


def _exact_render(case, seed):
    x = {k: v.double() for k, v in _render_inputs(case, seed).items()}
    B, C, W, H = case["frames"], case["views"], case["width"], case["height"]
    faces = torch.from_numpy(_mesh(case["subdiv"])[1]).to(DEV, torch.int64)
    albedo = case["albedo"]
    shaded = case["shading"] == "shaded" and albedo in ("vertexColor", "textured", "texturedBilinear")
    leaves = [x[k].requires_grad_() for k in ("verts", "colors", "texture", "sh")]
    verts, colors, texture, sh = leaves
    tri = verts[:, faces]
    fn = torch.linalg.cross(tri[:, :, 1] - tri[:, :, 0], tri[:, :, 2] - tri[:, :, 0])
    vn = torch.zeros_like(verts)
    for k in range(3):
        vn = vn.index_add(1, faces[:, k], fn)
    uv = torch.from_numpy(_texcoords(case["subdiv"])).to(DEV, torch.float64).view(-1, 3, 2)
    uv = torch.stack([uv[..., 0], 1.0 - uv[..., 1]], -1)
    bary, image = (torch.zeros(B, C, H * W, k, device=DEV, dtype=torch.float64) for k in (2, 3))
    total = 0.0
    for b in range(B):
        for c in range(C):
            E, K = x["extr"][b, 12 * c:12 * c + 12].view(3, 4), x["intr"][b, 9 * c:9 * c + 9].view(3, 3)
            o = -E[:, :3].T @ E[:, 3]
            pix, f = _visible(verts[b].detach(), faces, E, K, o, W, H)
            q = torch.stack([pix % W + 0.5, torch.div(pix, W, rounding_mode="floor") + 0.5, torch.ones_like(pix)], 1)
            ray = (torch.linalg.inv(K @ E[:, :3]) @ q.double().T).T
            ray = ray / ray.norm(dim=1, keepdim=True)
            p = tri[b, f]
            l0, l1 = _barycentrics(o, ray, p)
            l2 = 1 - l0 - l1
            lam = torch.stack([l0, l1, l2], 1)
            # the adjoint leaves barycentrics of grazing hits out
            n = torch.linalg.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]).detach()
            cut = ((ray * n).sum(1) / n.norm(dim=1)).abs() < 0.001
            lam = torch.where(cut[:, None], lam.detach(), lam)
            pn = (lam[..., None] * vn[b][faces[f]]).sum(1)
            pn = pn / pn.norm(dim=1, keepdim=True)
            pn = torch.where((pn * ray).sum(1, keepdim=True) > 0, -pn, pn)
            if albedo == "vertexColor":
                col = (lam[..., None] * colors[b][faces[f]]).sum(1)
            elif albedo == "texturedBilinear":
                t = case["texture"]
                col = _bilinear(texture[b], (lam[..., None] * uv[f]).sum(1) * t)
            elif albedo == "normal":
                col = (1 + pn) / 2
            elif albedo == "depth":
                col = ((lam[..., None] * p).sum(1) - o).norm(dim=1, keepdim=True).expand(-1, 3)
            else:  # the nearest-texel mode jumps at texel edges: no value in 64 bits
                col = torch.zeros_like(pn)
            if shaded:
                col = col * _light(sh[b, c], pn)
            bary[b, c, pix] = torch.stack([l0, l1], 1).detach()
            image[b, c, pix] = col.detach()
            if case["backward"]:
                g = x["grad"][b, c].reshape(-1, 3)[pix]
                total = total + (g * col).sum()
                # the target's image gradient moves the fragment (weights held)
                du, dv = _sobel(x["target"][b, c])
                P = (lam.detach()[..., None] * p).sum(1) @ (K @ E[:, :3]).T + K @ E[:, 3]
                gu = (g * du.reshape(-1, 3)[pix]).sum(1)
                gv = (g * dv.reshape(-1, 3)[pix]).sum(1)
                total = total - (gu * P[:, 0] / P[:, 2] + gv * P[:, 1] / P[:, 2]).sum()
    # a pixel centre within float rounding of an edge may take the neighbouring face: barycentrics (and with them the
    # position gradient) have a value in 64 bits only where such pixels are few, on large triangles of moderate images
    steady = max(W, H) <= 1024 and W * H > 25 * len(faces) // 2
    out = [bary.view(B, C, H, W, 2) if steady else None, None,
           None if albedo == "textured" else image.view(B, C, H, W, 3),
           vn.detach()[:, None].expand(B, C, -1, 3)]
    if not case["backward"]:
        return out
    if albedo == "textured":
        return out + [None] * 4
    grads = torch.autograd.grad(total, leaves, allow_unused=True)
    grads = [torch.zeros_like(v) if g is None else g for g, v in zip(grads, leaves)]
    return out + [grads[0] if steady and albedo == "vertexColor" else None] + grads[1:]


def _visible(v, faces, E, K, o, W, H):
    """(pixel, nearest face) of every covered pixel, by testing each triangle on its bounding box."""
    p = (v @ E[:, :3].T + E[:, 3]) @ K.T
    p = (p[:, :2] / p[:, 2:])[faces]
    lo = (p.amin(1) - 0.5).floor().clamp_min(0).long()
    hi = torch.minimum((p.amax(1) + 0.5).floor().long(), torch.tensor([W - 1, H - 1], device=DEV))
    ext = (hi - lo + 1).clamp_min(0)
    area = ext[:, 0] * ext[:, 1]
    best = torch.full((W * H,), math.inf, device=DEV, dtype=torch.float64)
    hits = []
    ends = area.cumsum(0)
    cuts = torch.searchsorted(ends, torch.arange(0, int(ends[-1]) + 1, 1 << 23, device=DEV)).tolist() + [len(area)]
    iP = torch.linalg.inv(K @ E[:, :3])
    for a, z in zip(cuts, cuts[1:]):
        n = area[a:z]
        if z <= a or not int(n.sum()):
            continue
        f = torch.repeat_interleave(torch.arange(a, z, device=DEV), n)
        k = torch.arange(len(f), device=DEV) - (n.cumsum(0) - n)[f - a]
        px, py = lo[f, 0] + k % ext[f, 0], lo[f, 1] + torch.div(k, ext[f, 0], rounding_mode="floor")
        ray = torch.stack([px + 0.5, py + 0.5, torch.ones_like(px)], 1).double() @ iP.T
        ray = ray / ray.norm(dim=1, keepdim=True)
        t3 = v[faces[f]]
        l0, l1, t = _barycentrics(o, ray, t3, True)
        ok = (l0 >= 0) & (l1 >= 0) & (l0 + l1 <= 1) & (t > 0)
        pix = (py * W + px)[ok]
        best.scatter_reduce_(0, pix, t[ok], "amin")
        hits.append((pix, f[ok], t[ok]))
    pix, f, t = (torch.cat(h) for h in zip(*hits))
    won = t <= best[pix]
    pix, f = pix[won], f[won]
    order = torch.argsort(pix * len(faces) + f)
    pix, f = pix[order], f[order]
    first = torch.ones_like(pix, dtype=torch.bool)
    first[1:] = pix[1:] != pix[:-1]
    return pix[first], f[first]


def _barycentrics(o, ray, p, depth=False):
    v0, v1, v2 = p[:, 0], p[:, 1], p[:, 2]
    n = torch.linalg.cross(v1 - v0, v2 - v0)
    t = ((v0 - o) * n).sum(1) / (ray * n).sum(1)
    x = o + t[:, None] * ray
    den = (n * n).sum(1)
    l0 = (n * torch.linalg.cross(v2 - v1, x - v1)).sum(1) / den
    l1 = (n * torch.linalg.cross(v0 - v2, x - v2)).sum(1) / den
    return (l0, l1, t) if depth else (l0, l1)


def _bilinear(tex, xy):
    s = xy - 0.5
    i = s.detach().floor()
    fx, fy = (s - i)[:, :1], (s - i)[:, 1:]
    x0, y0 = i[:, 0].long(), i[:, 1].long()
    at = lambda y, x: tex[y.clamp(0, tex.shape[0] - 1), x.clamp(0, tex.shape[1] - 1)]  # noqa: E731
    return (at(y0, x0) * (1 - fx) * (1 - fy) + at(y0, x0 + 1) * fx * (1 - fy) + at(y0 + 1, x0) * (1 - fx) * fy
            + at(y0 + 1, x0 + 1) * fx * fy)


def _light(sh, n):
    x, y, z = n.unbind(1)
    basis = torch.stack([torch.ones_like(x), y, z, x, x * y, z * y, 3 * z * z - 1, x * z, x * x - y * y], 1)
    return basis @ sh.view(3, 9).T


def _sobel(img, fs=2):
    """Image gradients with weights (i, j) / (i^2 + j^2) over (2 fs + 1)^2 taps, zero near the border."""
    H, W, _ = img.shape
    du, dv = torch.zeros_like(img), torch.zeros_like(img)
    m = fs + 1
    if H <= 2 * m or W <= 2 * m:
        return du, dv
    norm = 0.0
    for j in range(-fs, fs + 1):
        for i in range(-fs, fs + 1):
            if i or j:
                w = 1.0 / (i * i + j * j)
                part = img[m + j:H - m + j, m + i:W - m + i]
                du[m:H - m, m:W - m] += part * (i * w)
                dv[m:H - m, m:W - m] += part * (j * w)
                norm += abs(i * w)
    return du / norm, dv / norm


# ----------------------------------------------------------------------------
# uv
# ----------------------------------------------------------------------------
def _prepare_uv(case, seed):
    d, B, t = _Draws(seed), case["frames"], case["texture"]
    verts = _posed_mesh(case, d)
    ex, it = _cameras(1, [(64, 64)], B)
    eng = RendererEngine(_mesh(case["subdiv"])[1], _texcoords(case["subdiv"]), verts.shape[1], 1, 64, 64, "textured",
                         "shadeless", 2, 2, "normal")
    return dict(engine=eng, args=(verts, d.uniform(0, 1, *verts.shape), d.uniform(0, 1, B, t, t, 3), d.sh(B, 1), ex,
                                  it))


def _run_uv(s):
    out = s["engine"].forward(*s["args"])
    return [out[3], out[4]]


# ----------------------------------------------------------------------------
# deform
# ----------------------------------------------------------------------------
def _deform_inputs(case, seed):
    d, B = _Draws(seed), case["frames"]
    sc = _scene(case["subdiv"], case["nodes"])
    M, N = sc["graph"].n_nodes, sc["verts"].shape[0]
    return sc, dict(dofs=d.uniform(-0.5, 0.5, B, sc["skeleton"].n_dofs), dT=d.normal(0.01 * S.MM, B, M, 3),
                    dA=d.normal(0.05, B, M, 3), disp=d.normal(1.0, B, N, 3), gv=d.normal(1.0, B, N, 3),
                    gm=d.normal(1.0, B, 8, 3))


def _prepare_deform(case, seed):
    sc, x = _deform_inputs(case, seed)
    s = dict(skin=SkinningEngine(character(sc)), eg=EmbeddedGraphEngine(eg_data(sc), full_skinned_gradient=True),
             node_vertex=torch.from_numpy(sc["graph"].node_vertex).to(DEV),
             weights=torch.from_numpy(sc["skin_weights"]).to(DEV), **x)
    for k in ("dT", "dA", "disp"):
        s[k].requires_grad_()
    return s


def _run_deform(s):
    sT, sA, dq = s["skin"].pose2eg(s["dofs"], s["node_vertex"], s["weights"])
    sT.requires_grad_()
    sA.requires_grad_()
    v, n, m, g = EmbeddedGraphGpu(numberOfBatches=s["dT"].shape[0], deltaT=s["dT"], deltaR=s["dA"], skinnedT=sT,
                                  skinnedR=sA, displacements=s["disp"], engine=s["eg"]).getNode()
    gT, gA, gsT, gsA, gdisp = torch.autograd.grad([v, m], [s["dT"], s["dA"], sT, sA, s["disp"]], [s["gv"], s["gm"]])
    gdofs = s["skin"].pose2eg_backward(s["dofs"], s["node_vertex"], s["weights"], gsT, gsA)
    return [sT, sA, dq, v, n, m, g, gT, gA, gsT, gsA, gdisp, gdofs]


def _exact_deform(case, seed):
    sc, x = _deform_inputs(case, seed)
    x = {k: v.double() for k, v in x.items()}
    t64 = lambda a: torch.from_numpy(np.asarray(a)).to(DEV, torch.float64)  # noqa: E731
    dofs = x["dofs"].requires_grad_()
    g = sc["graph"]
    nv = torch.from_numpy(g.node_vertex).to(DEV).long()
    dq, _, _ = _kinematics(sc["skeleton"], dofs)
    idx = torch.from_numpy(sc["skin_index"]).to(DEV).long()[nv]
    R, T = _blend(dq, idx, t64(sc["skin_weights"])[nv])
    eul = torch.stack([torch.atan2(R[..., 2, 1], R[..., 2, 2]),
                       torch.atan2(-R[..., 2, 0], (R[..., 0, 0] ** 2 + R[..., 1, 0] ** 2).sqrt()),
                       torch.atan2(R[..., 1, 0], R[..., 0, 0])], -1)
    sT, sA = T.detach().requires_grad_(), eul.detach().requires_grad_()
    dT, dA, disp = (x[k].requires_grad_() for k in ("dT", "dA", "disp"))
    base = t64(sc["verts"])
    gb = base[nv]
    Rd, Rs = _euler(dA), _euler(sA)
    vi = torch.from_numpy(g.v2n_indices).to(DEV).long().view(-1, 4)
    w = t64(g.v2n_weights).view(-1, 4)
    u, v = disp, 0.0
    for k in range(4):
        i = vi[:, k]
        u = u + w[:, k:k + 1] * ((Rd[:, i] @ (base - gb[i])[None, ..., None])[..., 0] + gb[i] + dT[:, i])
    for k in range(4):
        i = vi[:, k]
        v = v + w[:, k:k + 1] * ((Rs[:, i] @ u[..., None])[..., 0] + sT[:, i])
    n = _mesh_normals(v.detach(), sc["faces"])
    mk = torch.from_numpy(sc["marker_node"]).to(DEV).long()
    mu = (Rd[:, mk] @ (t64(sc["markers"]) - gb[mk])[None, ..., None])[..., 0] + gb[mk] + dT[:, mk]
    m = (Rs[:, mk] @ mu[..., None])[..., 0] + sT[:, mk]
    node = (Rs @ (gb + dT)[..., None])[..., 0] + sT
    grads = torch.autograd.grad([v, m], [dT, dA, sT, sA, disp], [x["gv"], x["gm"]])
    gd, = torch.autograd.grad([T, eul], [dofs], [grads[2], grads[3]])
    return [sT, sA, None, v, n / n.norm(dim=-1, keepdim=True), m, node, *grads, gd]


def _euler(a):
    c, s = a.cos(), a.sin()
    one, zero = torch.ones_like(c[..., 0]), torch.zeros_like(c[..., 0])
    mat = lambda *e: torch.stack(e, -1).reshape(*one.shape, 3, 3)  # noqa: E731
    rx = mat(one, zero, zero, zero, c[..., 0], -s[..., 0], zero, s[..., 0], c[..., 0])
    ry = mat(c[..., 1], zero, s[..., 1], zero, one, zero, -s[..., 1], zero, c[..., 1])
    rz = mat(c[..., 2], -s[..., 2], zero, s[..., 2], c[..., 2], zero, zero, zero, one)
    return rz @ ry @ rx


def _mesh_normals(v, faces):
    f = torch.from_numpy(faces).to(DEV).long()
    t = v[:, f]
    fn = torch.linalg.cross(t[:, :, 1] - t[:, :, 0], t[:, :, 2] - t[:, :, 0])
    n = torch.zeros_like(v)
    for k in range(3):
        n.index_add_(1, f[:, k], fn)
    return n


def _kinematics(sk, dofs):
    """(dual quaternions [B,S,8], joint positions, joint axes) in 64 bits."""
    B = dofs.shape[0]
    R, t, rest = [], [], []
    off, axis = (torch.from_numpy(a).to(DEV, torch.float64) for a in (sk.offset, sk.axis))
    for j in range(sk.n_joints):
        x, y, z = axis[j]
        k = torch.stack([torch.zeros_like(x), -z, y, z, torch.zeros_like(x), -x, -y, x, torch.zeros_like(x)]).view(3, 3)
        th = dofs[:, j, None, None]
        local = torch.eye(3, device=DEV, dtype=torch.float64) + th.sin() * k + (1 - th.cos()) * (k @ k)
        p = int(sk.parent[j])
        R.append(local if p < 0 else R[p] @ local)
        t.append(off[j].expand(B, 3) if p < 0 else R[p] @ off[j] + t[p])
        rest.append(off[j] if p < 0 else rest[p] + off[j])
    dq = []
    for j in sk.skin_joint.tolist():
        q = _quaternion(R[j])
        tr = t[j] - (R[j] @ rest[j])
        tv = torch.cat([tr, torch.zeros_like(tr[:, :1])], 1)
        dq.append(torch.cat([q, 0.5 * _qmul(tv, q)], 1))
    ax = [(R[j] @ axis[j]) for j in range(sk.n_joints)]
    return torch.stack(dq, 1), torch.stack(t, 1), torch.stack(ax, 1)


def _qmul(p, q):
    pv, pw, qv, qw = p[..., :3], p[..., 3:], q[..., :3], q[..., 3:]
    return torch.cat([pw * qv + qw * pv + torch.linalg.cross(pv, qv), pw * qw - (pv * qv).sum(-1, keepdim=True)], -1)


def _quaternion(R):
    """(x, y, z, w) of rotation matrices, from the largest of the four components."""
    d = torch.stack([R[:, 0, 0], R[:, 1, 1], R[:, 2, 2]], 1)
    tr = d.sum(1)
    w = torch.stack([R[:, 2, 1] - R[:, 1, 2], R[:, 0, 2] - R[:, 2, 0], R[:, 1, 0] - R[:, 0, 1], 1 + tr], 1)
    cand = [w]
    for i in range(3):
        j, k = (i + 1) % 3, (i + 2) % 3
        e = [None] * 4
        e[i], e[j], e[k] = 1 + 2 * d[:, i] - tr, R[:, j, i] + R[:, i, j], R[:, k, i] + R[:, i, k]
        e[3] = R[:, k, j] - R[:, j, k]
        cand.append(torch.stack(e, 1))
    best = torch.where(tr > 0, torch.zeros_like(tr).long(), d.argmax(1) + 1)
    q = torch.stack(cand, 1)[torch.arange(len(R), device=DEV), best]
    return q / q.norm(dim=1, keepdim=True)


def _blended(dq, idx, w):
    """Sign-aligned sums of the vertices' dual quaternions, and each slot's aligned one."""
    q = dq[:, idx]
    sign = torch.where((q[..., :1, :4] * q[..., :4]).sum(-1, keepdim=True) < 0, -1.0, 1.0)
    q = q * sign
    return (w[..., None] * q).sum(-2), q


def _blend(dq, idx, w):
    b, _ = _blended(dq, idx, w)
    return _rigid(b / b[..., :4].norm(dim=-1, keepdim=True))


def _rigid(b):
    x, y, z, w = b[..., :4].unbind(-1)
    R = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w), 2 * (x * y + z * w),
                     1 - 2 * (x * x + z * z), 2 * (y * z - x * w), 2 * (x * z - y * w), 2 * (y * z + x * w),
                     1 - 2 * (x * x + y * y)], -1).reshape(*x.shape, 3, 3)
    conj = torch.cat([-b[..., :3], b[..., 3:4]], -1)
    return R, 2 * _qmul(b[..., 4:], conj)[..., :3]


# ----------------------------------------------------------------------------
# skin
# ----------------------------------------------------------------------------
def _skin_inputs(case, seed):
    d, B = _Draws(seed), case["frames"]
    sk, idx, w = _skeleton(case["subdiv"])
    _, faces, verts = _mesh(case["subdiv"])
    N = verts.shape[0]
    return sk, idx, verts, faces, dict(
        dofs=d.uniform(-0.5, 0.5, B, sk.n_dofs), weights=torch.from_numpy(w).to(DEV).repeat(B, 1, 1),
        disp=d.normal(1.0, B, N, 3), gv=d.normal(1.0, B, N, 3))


def _prepare_skin(case, seed):
    sk, idx, verts, faces, x = _skin_inputs(case, seed)
    sc = dict(skeleton=sk, verts=verts, faces=faces, skin_index=idx)
    for k in ("dofs", "weights", "disp"):
        x[k].requires_grad_()
    return dict(mode=case["mode"], engine=SkinningEngine(character(sc)), **x)


def _run_skin(s):
    if s["mode"] == "dq":
        out, leaves = dq_skinning_gpu(s["engine"], s["dofs"], s["weights"]), [s["dofs"], s["weights"]]
    else:
        out = lb_skinning_gpu(s["engine"], s["dofs"], s["weights"], s["disp"])
        leaves = [s["dofs"], s["weights"], s["disp"]]
    return [*out, *torch.autograd.grad(out[0], leaves, s["gv"])]


def _exact_skin(case, seed):
    sk, idx, verts, faces, x = _skin_inputs(case, seed)
    x = {k: v.double() for k, v in x.items()}
    t64 = lambda a: torch.from_numpy(np.asarray(a)).to(DEV, torch.float64)  # noqa: E731
    idx = torch.from_numpy(idx).to(DEV).long()
    dq, gp, ga = _kinematics(sk, x["dofs"])
    base, w, g = t64(verts), x["weights"], x["gv"]
    n0 = _mesh_normals(base[None], faces)[0]
    n0 = n0 / n0.norm(dim=1, keepdim=True)
    Rj, Tj = _rigid(dq)
    if case["mode"] == "dq":
        b, q = _blended(dq, idx, w)
        R, T = _rigid(b / b[..., :4].norm(dim=-1, keepdim=True))
        v = (R @ base[None, ..., None])[..., 0] + T
    else:
        R, T = (w[..., None, None] * Rj[:, idx]).sum(2), (w[..., None] * Tj[:, idx]).sum(2)
        v = (R @ (base + x["disp"])[..., None])[..., 0] + T
    n = (R @ n0[None, ..., None])[..., 0]
    if case["mode"] == "dq":
        n = n / n.norm(dim=-1, keepdim=True)
    # linearised joint gradient: every joint turns what hangs below it about its axis
    below = torch.zeros(sk.n_joints, sk.n_skin, device=DEV, dtype=torch.float64)
    for s, j in enumerate(sk.skin_joint.tolist()):
        while j >= 0:
            below[j, s] = 1.0
            j = int(sk.parent[j])
    mom = torch.zeros(v.shape[0], sk.n_skin, 6, device=DEV, dtype=torch.float64)
    vg = torch.cat([torch.linalg.cross(v, g), g], -1)
    for k in range(idx.shape[1]):
        mom.index_add_(1, idx[:, k], w[:, :, k:k + 1] * vg)
    m = below @ mom
    gd = (ga * (m[..., :3] - torch.linalg.cross(gp, m[..., 3:]))).sum(-1)
    tr = dq if case["mode"] == "dq" else torch.cat([Rj.reshape(*Rj.shape[:2], 9), Tj], -1)
    out = [v, n, gp, ga, None if case["mode"] == "dq" else tr, w]
    if case["mode"] == "dq":
        return out + [gd, _dq_weight_gradient(b, q, base, g)]
    # the weight and displacement gradients read transform k for slot k, without the displacement
    gw = torch.stack([(((Rj[:, k, None] @ base[None, ..., None])[..., 0] + Tj[:, k, None]) * g).sum(-1)
                      for k in range(idx.shape[1])], -1)
    w0 = torch.where(w[:1] < 1e-4, torch.zeros_like(w[:1]), w[:1])
    gdisp = sum(w0[..., k:k + 1] * (Rj[:, k, None].transpose(-1, -2) @ g[..., None])[..., 0]
                for k in range(idx.shape[1]))
    return out + [gd, gw, gdisp]


def _dq_weight_gradient(b, q, base, g):
    """The op's weight gradient, whose rotation Jacobian adds the point's z where it should multiply by it."""
    s = b[..., :4].norm(dim=-1, keepdim=True)
    u = b / s
    d = (q - u[..., None, :] * (u[..., None, :4] * q[..., :4]).sum(-1, keepdim=True)) / s[..., None]
    x, y, z, w = u[..., :4].unbind(-1)
    o = torch.zeros_like(x)
    rows = [((o, -4 * y, -4 * z, o), (2 * y, 2 * x, -2 * w, -2 * z), (2 * z, 2 * w, 2 * x, 2 * y)),
            ((2 * y, 2 * x, 2 * w, 2 * z), (-4 * x, o, -4 * z, o), (-2 * w, 2 * z, 2 * y, -2 * x)),
            ((2 * z, -2 * w, 2 * x, -2 * y), (2 * w, 2 * z, 2 * y, 2 * x), (-4 * x, -4 * y, o, o))]
    jac = torch.stack([torch.stack([r[0][c] * base[:, 0] + r[1][c] * base[:, 1] + r[2][c] + base[:, 2]
                                    for c in range(4)], -1) for r in rows], -2)
    rot = (jac[..., None, :, :] @ d[..., :4, None])[..., 0]
    conj = lambda p: torch.cat([-p[..., :3], p[..., 3:4]], -1)  # noqa: E731
    tr = 2 * (_qmul(d[..., 4:], conj(u)[..., None, :]) + _qmul(u[..., None, 4:].expand_as(d[..., 4:]),
                                                                 conj(d)))[..., :3]
    return ((rot + tr) * g[..., None, :]).sum(-1)


# ----------------------------------------------------------------------------
# sil
# ----------------------------------------------------------------------------
def _sil_inputs(case, seed):
    d, B, C, W, H = _Draws(seed), case["frames"], case["views"], case["width"], case["height"]
    verts = _posed_mesh(case, d)
    ex, it = _cameras(C, _sizes(case), B)
    normals = _mesh_normals(verts, _mesh(case["subdiv"])[1])
    normals = normals / normals.norm(dim=-1, keepdim=True)
    # the op names dimension 2 of the distance image U and dimension 3 V: [B, C, W, H]
    dt = torch.stack(d.masks(B, _sizes(case)), 1).reshape(B, C, W, H)
    return dict(verts=verts, normals=normals, extr=ex, intr=it, dt=dt,
                crops=torch.from_numpy(S.identity_crops(B, C, W, H)).to(DEV), g=d.normal(1.0, B, C, verts.shape[1]),
                g1=d.normal(1.0, B, C, H, W, 2))


def _prepare_sil(case, seed):
    x = _sil_inputs(case, seed)
    x["verts"].requires_grad_()
    return dict(size=(case["width"], case["height"]), engine=SilhouetteEngine(),
                boundary=MeshBoundaryEngine(_mesh(case["subdiv"])[1], x["verts"].shape[1]), **x)


def _run_sil(s):
    p = CameraProjectionGpu(True, s["verts"], None, s["extr"], s["intr"]).getNode()
    with torch.no_grad():
        n = CameraProjectionGpu(False, s["verts"], s["normals"], s["extr"], s["intr"]).getNode()
        isb = s["boundary"].forward(s["verts"], s["extr"], s["intr"], *s["size"], points_image_space=p)
    res, res1, dtg, cid = MultiViewSilhouetteLossGpu(p, n, isb, s["dt"], s["crops"], engine=s["engine"]).getNode()
    grad, = torch.autograd.grad([res, res1], [s["verts"]], [s["g"], s["g1"]])
    return [p, n, isb, res, res1, dtg, cid, grad]


def _exact_sil(case, seed):
    x = {k: v.double() for k, v in _sil_inputs(case, seed).items() if k in ("verts", "normals", "extr", "intr")}
    B, C = case["frames"], case["views"]
    E, K = x["extr"].view(B, C, 3, 4), x["intr"].view(B, C, 3, 3)
    cam = (E[..., :3] @ x["verts"][:, None].transpose(-1, -2) + E[..., 3:])
    image = lambda c: (lambda h: (h[:, :, :2] / h[:, :, 2:]).transpose(-1, -2))(K @ c)  # noqa: E731
    p = image(cam)
    n = image(cam + E[..., :3] @ x["normals"][:, None].transpose(-1, -2)) - p
    # the losses step at whole pixels and whole vertices: no value in 64 bits
    return [p, n / n.norm(dim=-1, keepdim=True)] + [None] * 6


# ----------------------------------------------------------------------------
# images
# ----------------------------------------------------------------------------
def _images_inputs(case, seed):
    d, shape = _Draws(seed), (1, case["images"], case["height"], case["width"])
    face = torch.randint(-1, 3, shape, device=DEV, generator=d.g, dtype=torch.int32)
    return dict(image=d.image(*shape, 3), render=d.uniform(0, 1, *shape, 3), face=face, size=case["size"])


def _run_images(s):
    smooth = smooth_image(s["image"], s["size"], 0.0, 0.5 * s["size"])
    return [smooth, *image_l1_loss(s["render"], s["image"], s["face"])]


def _exact_images(case, seed):
    x = _images_inputs(case, seed)
    k = torch.arange(-case["size"], case["size"] + 1, device=DEV, dtype=torch.float64)
    w = torch.exp(-0.5 * (k / (0.5 * case["size"])) ** 2)
    w = w / w.sum()
    img = x["image"].double()[0].permute(0, 3, 1, 2)
    for dim in (2, 3):
        pad = torch.nn.functional.pad(img, (0, 0, case["size"], case["size"]) if dim == 2 else
                                      (case["size"], case["size"], 0, 0))
        n = img.shape[dim]
        img = sum(w[i] * pad.narrow(dim, i, n) for i in range(len(w)))
    r, t = x["render"] * 255.0, x["image"] * 255.0  # each product rounded on its own
    d = (r.double() - t.double()) * (x["face"] >= 0)[..., None]
    count = torch.count_nonzero(d)
    return [img.permute(0, 2, 3, 1)[None], (d.abs().sum() / count)[None], d.sign() * 255.0 / count]


# ----------------------------------------------------------------------------
# chain
# ----------------------------------------------------------------------------
def _prepare_chain(case, seed):
    d, B, C = _Draws(seed), case["frames"], case["views"]
    sc, sizes = _scene(case["subdiv"], case["nodes"]), _sizes(case)
    M, N, P = sc["graph"].n_nodes, sc["verts"].shape[0], sum(w * h for w, h in sizes)
    mixed = len(set(sizes)) > 1
    W, H = [w for w, _ in sizes], [h for _, h in sizes]
    img = (B, P) if mixed else (B, C, H[0], W[0])
    ex, it = _cameras(C, sizes, B)
    crops = np.stack([np.array([0, 0, 1, 0, 0, w, h], np.float32) for w, h in sizes])
    z = lambda *s: np.zeros(s, np.float32)  # noqa: E731
    sc.update(dofs=z(B, sc["skeleton"].n_dofs), dT=z(B, M, 3), dA=z(B, M, 3), disp=z(B, N, 3), colors=z(B, N, 3),
              texture=z(B, 16, 16, 3), sh=z(B, C, 27), extr=ex.cpu().numpy(), intr=it.cpu().numpy(),
              target=z(*img, 3), dt=np.zeros(img, np.uint8), crops=np.tile(crops[None], (B, 1, 1)),
              texcoords=_texcoords(case["subdiv"]))
    ch = DeformRenderChain(sc, torch.device(DEV), B, C, W if mixed else W[0], H if mixed else H[0],
                           gradient_parity=case["parity"], deformation=case["deformation"])
    # this step's inputs, as a loader writes them into the chain's buffers
    i = ch.inp
    i["dofs"].copy_(d.uniform(-0.5, 0.5, *i["dofs"].shape))
    i["dT"].copy_(d.normal(0.01 * S.MM, B, M, 3))
    i["dA"].copy_(d.normal(0.05, B, M, 3))
    i["colors"].copy_(d.uniform(0, 1, 1, N, 3))
    i["sh"].copy_(d.sh(B, C))
    i["target"].copy_(d.image(*img, 3))
    i["dt"].copy_(torch.cat([m.reshape(B, -1) for m in d.masks(B, sizes)], 1).view(img))
    ch.step()
    torch.cuda.synchronize()
    return dict(chain=ch, graph=ch.capture_step())


def _run_chain(s):
    s["graph"].replay()
    ch = s["chain"]
    keys = ["v", "face", "render", "bary", "isb", "res", "gcol", "gdofs"] + (["gT", "gA"] if ch.M else [])
    return [ch.loss] + [ch.buf[k] for k in keys]


# ----------------------------------------------------------------------------
# entry points
# ----------------------------------------------------------------------------
def prepare(case, seed):
    if case["kind"] == "images":
        return _images_inputs(case, seed)
    return {"render": _prepare_render, "uv": _prepare_uv, "deform": _prepare_deform, "skin": _prepare_skin,
            "sil": _prepare_sil, "chain": _prepare_chain}[case["kind"]](case, seed) | {"kind": case["kind"]}


def run(state):
    return {"render": _run_render, "uv": _run_uv, "deform": _run_deform, "skin": _run_skin, "sil": _run_sil,
            "images": _run_images, "chain": _run_chain}[state.get("kind", "images")](state)


def exact(case, seed):
    """64-bit values; none for the UV maps (their texel table is defined by a float ray test) and the whole chain."""
    f = {"render": _exact_render, "deform": _exact_deform, "skin": _exact_skin, "sil": _exact_sil,
         "images": _exact_images}.get(case["kind"])
    if f is None or case["kind"] == "render" and case["frames"] * case["views"] * case["subdiv"] > 400:
        return None
    return f(case, seed)


def work(case):
    """Bytes: inputs read once and outputs written once.  Flops: of the arithmetic the outputs cannot do without."""
    k = case["kind"]
    if k == "images":
        px = case["images"] * case["width"] * case["height"]
        return dict(bytes=px * (12 + 12 + 12 + 4 + 12), flops=px * 3 * (4 * (2 * case["size"] + 1) + 4))
    B, N = case["frames"], 10 * 4 ** case["subdiv"] + 2
    F = 2 * N - 4
    if k == "uv":
        t = case["texture"] ** 2
        return dict(bytes=12 * F + B * (24 * N + 12 * t) + 12 * t, flops=B * (30 * t + 20 * F))
    if k == "deform":
        M = min(case["nodes"], N // 4)
        return dict(bytes=B * (N * 84 + M * 120) + 92 * N, flops=B * (N * 4 * 120 + M * 600))
    if k == "skin":
        return dict(bytes=B * N * (24 + 36 + 16 * 3) + N * 40, flops=B * N * 4 * 90)
    C, px = case["views"], B * sum(w * h for w, h in _sizes(case))
    if k == "sil":
        return dict(bytes=px * (1 + 8 + 4 + 8) + B * C * N * (8 + 8 + 1 + 4 + 8 + 4) + B * N * 36 + 12 * F,
                    flops=B * C * N * 120)
    if k == "render":
        tex = 12 * case["texture"] ** 2 * B if case["albedo"].startswith("textured") else 12 * B * N
        fwd = dict(bytes=px * 24 + 12 * F + B * N * 12 * (1 + C) + tex, flops=px * 60 + B * C * F * 60)
        if not case["backward"]:
            return fwd
        return dict(bytes=fwd["bytes"] + px * (12 + 12) + B * N * 12 + tex, flops=fwd["flops"] + px * 300)
    return dict(bytes=37 * px + B * (136 * N + 24 * F), flops=px * 360 + B * C * F * 120)
