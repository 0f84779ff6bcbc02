// Forward rasterizer: camera set-up, vertex normals, triangle set-up with
// screen-tile binning, spill-over raster and the per-tile visibility resolve
// fused with barycentric / face-id / albedo / SH shading output.
//
// Reference behaviour (CudaRenderer/cpp/src/Renderer/CUDABasedRasterization.cu):
// one thread per (view, triangle) loops over the triangle's pixel bbox twice,
// first an int atomicMin on the quantised depth, then a racy write of every
// triangle whose depth equals the minimum.  Here each pixel is owned by one
// thread of its tile's CTA: the triangles binned to the tile are staged in
// shared memory and every thread keeps the minimum (depth_q, triangle) of its
// pixel in registers, so the common path has no atomics and the winner among
// equal depths is deterministic (smallest triangle id).  Triangles beyond the
// tile's bin capacity go through a spill list resolved with a 64-bit packed
// atomicMin and merged afterwards.
#include <algorithm>

#include "renderer.cuh"

namespace hc {

// ---------------------------------------------------------------------------
// camera set-up: one thread per view (reference initializeCamerasDevice,
// CUDABasedRasterization.cu:23-67, which runs <<<1,1>>> per frame)
// ---------------------------------------------------------------------------
__global__ void k_view_setup(int V, int C, const float* __restrict__ extr, const float* __restrict__ intr,
                             const CamLayout* __restrict__ layout, long long P_frame, long long T_frame,
                             long long Tb_frame, ViewCam* __restrict__ cams, int view_blocks, FillRuns fills) {
    if ((int)blockIdx.x >= view_blocks) {
        fill_runs(fills, (blockIdx.x - view_blocks) * (long long)blockDim.x + threadIdx.x,
                  (gridDim.x - view_blocks) * (long long)blockDim.x);
        return;
    }
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= V) return;
    {
        const CamLayout L = layout[v % C];
        const long long b = v / C;
        ViewCam& c = cams[v];
        c.W = L.W;
        c.H = L.H;
        c.tiles_x = L.tiles_x;
        c.tiles_x_b = L.tiles_x_b;
        c.fd_tiles_x = L.fd_tiles_x;
        c.fd_tiles_x_b = L.fd_tiles_x_b;
        c.pix_base = b * P_frame + L.pix;
        c.tile_base = b * T_frame + L.tile;
        c.tile_base_b = b * Tb_frame + L.tile_b;
    }
    const float* e = extr + 12 * (long long)v;
    const float* k = intr + 9 * (long long)v;
    M44 E, K;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        E.e[i] = (i % 5 == 0) ? 1.f : 0.f;
        K.e[i] = (i % 5 == 0) ? 1.f : 0.f;
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        K.e[4 * r + 0] = k[3 * r + 0];
        K.e[4 * r + 1] = k[3 * r + 1];
        K.e[4 * r + 2] = k[3 * r + 2];
        K.e[4 * r + 3] = 0.f;
        E.e[4 * r + 0] = e[4 * r + 0];
        E.e[4 * r + 1] = e[4 * r + 1];
        E.e[4 * r + 2] = e[4 * r + 2];
        E.e[4 * r + 3] = e[4 * r + 3];
    }
    const M44 invE = inverse44(E);
    const M44 invP = inverse44(mul44(K, E));
    ViewCam& c = cams[v];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        c.invP[i] = invP.e[i];
        c.invE[i] = invE.e[i];
    }
#pragma unroll
    for (int i = 0; i < 12; ++i) c.ext[i] = e[i];
#pragma unroll
    for (int i = 0; i < 9; ++i) c.intr[i] = k[i];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
#pragma unroll
        for (int cc = 0; cc < 3; ++cc)
            c.KE[3 * r + cc] = k[3 * r + 0] * e[cc] + k[3 * r + 1] * e[4 + cc] + k[3 * r + 2] * e[8 + cc];
        c.Kt[r] = k[3 * r + 0] * e[3] + k[3 * r + 1] * e[7] + k[3 * r + 2] * e[11];
    }
    // camera centre: last column of inv(E), dehomogenised
    float4 o = make_float4(invE.e[3], invE.e[7], invE.e[11], invE.e[15]);
    const float w = o.w;
    o.x /= w;
    o.y /= w;
    o.z /= w;
    c.ro[0] = o.x;
    c.ro[1] = o.y;
    c.ro[2] = o.z;
    c.ro_s[0] = o.x / 1000.f;
    c.ro_s[1] = o.y / 1000.f;
    c.ro_s[2] = o.z / 1000.f;
}

// ---------------------------------------------------------------------------
// a frame's mesh:
// - vertex normals: unnormalised sum of incident face normals, in increasing
//   face order (reference renderFaceNormalDevice / renderVertexNormalDevice,
//   CUDABasedRasterization.cu:122-174, computed once per frame and written for
//   every camera of the [B,C,N,3] output).  Bound by their gathers (FanFace).
// - per-frame triangle constants
// - per-view vertex projection (reference projectVerticesDevice,
//   CUDABasedRasterization.cu:98-115): once per (view, vertex) instead of three
//   times per (view, triangle); the same function, so the same values
// One launch for the three (FrameSetup): with the camera set-up and the fills,
// 8 launches and 13.8 us became 2 launches and 6.1 us (one 512^2 view of 20,480
// triangles).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kSetupThreads) k_frame_setup(FrameSetup S) {
    unsigned blk = blockIdx.x;
    if (blk < S.normal_blocks) {
        const long long i = blk * (long long)blockDim.x + threadIdx.x;
        if (i >= (long long)S.B * S.N) return;
        const int b = (int)(i / S.N);
        const int v = (int)(i % S.N);
        const float3 s = fan_normal(S.verts + (long long)b * S.N * 3, S.fan, S.vf_id[v], v);
        for (int c = 0; c < S.C; ++c) st3(S.vnormal + (((long long)b * S.C + c) * S.N + v) * 3, s);
        if (S.unit) {
            const float3 u = unit_or_zero<false>(s);
            S.unit[i] = make_float4(u.x, u.y, u.z, 0.f);
        }
        return;
    }
    blk -= S.normal_blocks;
    if (blk < S.tri_blocks) {
        const long long i = blk * (long long)blockDim.x + threadIdx.x;
        if (i >= (long long)S.B * S.F) return;
        const int b = (int)(i / S.F);
        const int f = (int)(i % S.F);
        const float* P = S.verts + (long long)b * S.N * 3;
        const int3 id = S.faces[f];
        const float3 s0 = ld3(P + 3 * id.x) / 1000.f;
        const float3 s1 = ld3(P + 3 * id.y) / 1000.f;
        const float3 s2 = ld3(P + 3 * id.z) / 1000.f;
        const float3 n = cross(s1 - s0, s2 - s0);
        TriFrame t;
        t.a = make_float4(s0.x, s0.y, s0.z, n.x);
        t.b = make_float4(s1.x, s1.y, s1.z, n.y);
        t.c = make_float4(s2.x, s2.y, s2.z, n.z);
        S.tri[i] = t;
        return;
    }
    blk -= S.tri_blocks;
    if (blk < S.project_blocks) {
        const long long i = blk * (long long)blockDim.x + threadIdx.x;
        if (i >= (long long)S.B * S.C * S.N) return;
        const int view = (int)(i / S.N), v = (int)(i % S.N);
        const ViewCam& cam = S.cams[view];
        const float3 p = project_point(cam.ext, cam.intr, ld3(S.verts + ((long long)(view / S.C) * S.N + v) * 3));
        S.proj[i] = make_float4(p.x, p.y, p.z, 0.f);
        return;
    }
    blk -= S.project_blocks;
    const unsigned first = S.normal_blocks + S.tri_blocks + S.project_blocks;
    fill_runs(S.fills, blk * (long long)blockDim.x + threadIdx.x, (gridDim.x - first) * (long long)blockDim.x);
}

// ---------------------------------------------------------------------------
// per-view triangle set-up and screen-tile binning
//
// The pixel bbox is the reference's projectFacesDevice (CUDABasedRasterization.cu:
// 184-208): projected vertex extent +-0.5 px, clamped to the image, truncated to
// int.  Each (view, triangle) appends itself to every tile its bbox touches
// and its footprint reaches, taking a slot with one atomicAdd on the tile's
// counter; entries beyond the tile's capacity go to the spill list.
// ---------------------------------------------------------------------------
// Bound by instruction issue (73 % of the cycles) with the counters' round trips
// behind it.  Testing the box tile by tile, one counter at a time -> rows
// (TileRows), two counters at a time: 4 frames x 8 views of 81,920 triangles at
// 1024^2, 8-px tiles, 340 -> 267 us; 2 x 4 views of large triangles 162 -> 84.
// kBinSmall of 4: 439 us, 9: 304, 16: 267, 30: 266.
constexpr int kBinSmall = 16;  // tiles of a box that a thread bins on its own

// Where a (tile, triangle) pair goes once it has a slot in the tile's bin:
// the bin itself, or beyond the bin's capacity the spill list (the first
// overflowing pair of a tile claims and clears the tile's spill key block).
struct BinSink {
    int TS, cap;
    int2* tile_state;
    int* bins;
    int2* spill;  // (tile of the call, triangle)
    long long spill_cap;
    unsigned long long* spill_keys;
    int spill_tile_cap;
    RasterStats* stats;

    __device__ __forceinline__ int place(int slot, long long key, int f) const {
        if (slot < cap) {
            bins[key * cap + slot] = f;
            return 1;
        }
        if (slot == cap) {
            const int ks = atomicAdd(&stats->spill_tiles, 1);
            if (ks < spill_tile_cap) {
                unsigned long long* kp = spill_keys + (long long)ks * TS * TS;
                for (int p = 0; p < TS * TS; ++p) kp[p] = ~0ull;
                tile_state[key].y = ks + 1;
            } else {
                atomicOr(&stats->overflow, 2);
            }
        }
        const unsigned long long si = atomicAdd(&stats->spilled, 1ull);
        if ((long long)si < spill_cap) {
            spill[si] = make_int2((int)key, f);
        } else {
            atomicOr(&stats->overflow, 1);
        }
        return 0;
    }
};

__global__ void __launch_bounds__(256, 6) k_bin(int V, int C, int F, int N, int TS, int ts_shift, int cap,
                      const int3* __restrict__ faces, const float4* __restrict__ proj,
                      const ViewCam* __restrict__ cams, const TriFrame* __restrict__ tri_frame,
                      TriView* __restrict__ tri_view, int2* __restrict__ tile_state, int* __restrict__ bins,
                      int2* __restrict__ spill, long long spill_cap, unsigned long long* __restrict__ spill_keys,
                      int spill_tile_cap, RasterStats* __restrict__ stats) {
    // grid (triangle blocks, views): no 64-bit division per thread
    const int fi = blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = fi < F;
    const int view = blockIdx.y;
    const long long i = (long long)view * F + fi;
    int f = 0;
    int x0 = 0, x1 = -1, y0 = 0, y1 = -1;
    // the view is the block's (grid y), so its image and tile grid are the same in every lane
    const ViewCam& cam = cams[view];
    const int W = cam.W, H = cam.H, tiles_x = cam.tiles_x;
    const long long tile_base = cam.tile_base;
    TileRows rows;
    if (live) {
        f = fi;
        const int b = view / C;
        const int3 id = faces[f];
        const float4* PV = proj + (long long)view * N;
        const float4 q0 = PV[id.x], q1 = PV[id.y], q2 = PV[id.z];
        const float3 p0 = make_float3(q0.x, q0.y, q0.z), p1 = make_float3(q1.x, q1.y, q1.z),
                     p2 = make_float3(q2.x, q2.y, q2.z);
        x0 = (int)fmaxf(fminf(p0.x, fminf(p1.x, p2.x)) - 0.5f, 0.f);
        y0 = (int)fmaxf(fminf(p0.y, fminf(p1.y, p2.y)) - 0.5f, 0.f);
        x1 = (int)fminf(fmaxf(p0.x, fmaxf(p1.x, p2.x)) + 0.5f, (float)(W - 1));
        y1 = (int)fminf(fmaxf(p0.y, fmaxf(p1.y, p2.y)) + 0.5f, (float)(H - 1));
        const TriS T = tri_from(tri_frame[(long long)b * F + f]);
        const float3 ro_s = make_float3(cam.ro_s[0], cam.ro_s[1], cam.ro_s[2]);
        TriView tv;
        tv.num = dot(T.s0, T.n) - dot(ro_s, T.n);
        // x1/y1 can be negative for triangles left of / above the image
        // (empty bbox); store them clamped to -1 so the 16-bit packing keeps
        // the bbox empty.
        // x0/y0 beyond the image also mean an empty bbox (x1 <= W-1); clamp
        // them to W/H so they fit the 16-bit field.
        const int cx1 = max(x1, -1), cy1 = max(y1, -1);
        const int cx0 = min(x0, W), cy0 = min(y0, H);
        tv.x01 = (cx0 & 0xffff) | (cx1 << 16);
        tv.y01 = (cy0 & 0xffff) | (cy1 << 16);
        const Footprint fp = footprint(p0, p1, p2);
        rows = TileRows(fp);
        // the tile resolve copies this record as it is (no vertex gathers there)
        tv.e01 = make_float4(fp.a[0], fp.b[0], fp.a[1], fp.b[1]);
        tv.e2c = make_float4(fp.a[2], fp.b[2], fp.c[0], fp.c[1]);
        tv.c2 = fp.c[2];
        tri_view[i] = tv;
    }
    const bool nonempty = live && x1 >= x0 && y1 >= y0;
    int tx0 = 0, tx1 = -1, ty0 = 0, ty1 = -1;
    if (nonempty) {
        tx0 = x0 >> ts_shift;  // TS = 2^ts_shift; the box is non-empty, so x0 <= x1 are >= 0
        tx1 = x1 >> ts_shift;
        ty0 = y0 >> ts_shift;
        ty1 = y1 >> ts_shift;
    }
    const int ntx = tx1 - tx0 + 1;
    const int nt = nonempty ? ntx * (ty1 - ty0 + 1) : 0;
    const bool big = nt > kBinSmall;
    BinSink sink{TS, cap, tile_state, bins, spill, spill_cap, spill_keys, spill_tile_cap, stats};
    unsigned long long nbinned = 0;
    const unsigned lane = threadIdx.x & 31;
    // boxes of up to kBinSmall tiles: each lane finds the tiles of its own box that
    // the footprint reaches, then takes their slots, two counters in flight at once
    // (a slot's number is a round trip to L2)
    unsigned reached = 0u;
    if (!big && nt > 0) reached = nt == 1 ? 1u : rows.tiles(ts_shift, x0, x1, y0, y1);
    const float rn = __fdividef(1.f, (float)ntx);
    while (reached) {
        int tile[2], slot[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            slot[j] = -1;
            if (!reached) continue;
            const int k = __ffs(reached) - 1, r = (int)((k + 0.5f) * rn);
            reached &= reached - 1u;
            tile[j] = (ty0 + r) * tiles_x + tx0 + (k - r * ntx);
            slot[j] = atomicAdd(&tile_state[tile_base + tile[j]].x, 1);
        }
#pragma unroll
        for (int j = 0; j < 2; ++j)
            if (slot[j] >= 0) nbinned += sink.place(slot[j], tile_base + tile[j], f);
    }
    // larger boxes: the warp takes them one at a time
    unsigned pending = __ballot_sync(0xffffffffu, big);
    while (pending) {
        const int src = __ffs(pending) - 1;
        pending &= pending - 1;
        const int qf = __shfl_sync(0xffffffffu, f, src);
        const int qx0 = __shfl_sync(0xffffffffu, x0, src), qx1 = __shfl_sync(0xffffffffu, x1, src);
        const int qy0 = __shfl_sync(0xffffffffu, y0, src), qy1 = __shfl_sync(0xffffffffu, y1, src);
        warp_tiles(rows.from_lane(src), ts_shift, qx0, qx1, qy0, qy1, (int)lane, [&](int tx, int ty) {
            const int tile = ty * tiles_x + tx;
            nbinned += sink.place(atomicAdd(&tile_state[tile_base + tile].x, 1), tile_base + tile, qf);
        });
    }
    // one counter update per warp
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) nbinned += __shfl_xor_sync(0xffffffffu, nbinned, o);
    if (lane == 0 && nbinned) atomicAdd(&stats->binned, nbinned);
}

__device__ __forceinline__ void unpack_bbox(const TriView& tv, int& x0, int& x1, int& y0, int& y1) {
    x0 = tv.x01 & 0xffff;
    x1 = tv.x01 >> 16;
    y0 = tv.y01 & 0xffff;
    y1 = tv.y01 >> 16;
}

// ---------------------------------------------------------------------------
// spill raster: (view, tile, triangle) items beyond the bin capacity, one
// thread each, 64-bit packed atomicMin per pixel of tile x bbox.  With
// `count_depth` set (diagnostics) the pass instead counts, per pixel, the
// spilled triangles that reach the final depth.
// ---------------------------------------------------------------------------
__global__ void k_spill(int C, int F, int TS, long long T_frame, const int* __restrict__ tile_cam,
                        const ViewCam* __restrict__ cams, const TriFrame* __restrict__ tri_frame,
                        const TriView* __restrict__ tri_view, const int2* __restrict__ tile_state,
                        const int2* __restrict__ spill, long long spill_cap, int spill_tile_cap,
                        unsigned long long* __restrict__ spill_keys, const RasterStats* __restrict__ stats,
                        const int* __restrict__ count_depth, int* __restrict__ tie_out) {
    // one warp per spilled (tile, triangle) entry, its lanes over the pixels
    // of the triangle's box in the tile (the per-pixel atomic minimum does
    // not depend on the order)
    const long long n = min((long long)stats->spilled, spill_cap);
    const int lane = threadIdx.x & 31;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long i = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5; i < n; i += nwarps) {
        const int2 it = spill[i];
        const long long g = it.x;
        const int f = it.y;
        const int view = (int)(g / T_frame) * C + tile_cam[g % T_frame];
        const ViewCam& cam = cams[view];
        const int tile = (int)(g - cam.tile_base);
        const int ks = tile_state[g].y - 1;
        if (ks < 0 || ks >= spill_tile_cap) continue;
        const int W = cam.W, H = cam.H, tiles_x = cam.tiles_x;
        const TriView tv = tri_view[(long long)view * F + f];
        const TriS Tr = tri_from(tri_frame[(long long)(view / C) * F + f]);
        const float3 ro_s = make_float3(cam.ro_s[0], cam.ro_s[1], cam.ro_s[2]);
        int x0, x1, y0, y1;
        unpack_bbox(tv, x0, x1, y0, y1);
        const int tx = tile % tiles_x, ty = tile / tiles_x;
        const int px0 = max(x0, tx * TS), px1 = min(x1, min(tx * TS + TS - 1, W - 1));
        const int py0 = max(y0, ty * TS), py1 = min(y1, min(ty * TS + TS - 1, H - 1));
        const int bw = px1 - px0 + 1, bh = py1 - py0 + 1;
        if (bw <= 0 || bh <= 0) continue;
        for (int q = lane; q < bw * bh; q += 32) {
            {
                const int px = px0 + q % bw, py = py0 + q / bw;
                const float3 dir = pixel_ray<false>(cam, px, py);
                int dq;
                float a, b;
                if (!raster_hit(ro_s, dir, Tr, tv.num, dq, a, b)) continue;
                const int local = (py - ty * TS) * TS + (px - tx * TS);
                if (count_depth) {
                    const long long pix = cam.pix_base + (long long)py * W + px;
                    if (dq == count_depth[pix]) atomicAdd(&tie_out[pix], 1);
                } else {
                    const unsigned long long key = ((unsigned long long)(unsigned)dq << 32) | (unsigned)f;
                    atomicMin(&spill_keys[(long long)ks * TS * TS + local], key);
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// tile resolve + shading
// ---------------------------------------------------------------------------
struct ShadeArgs {
    int B, C, N, F;
    int albedo, shading;
    const int3* faces;
    const float* texcoords;
    const float* verts;
    const float* colors;
    const float* texture;
    int tex_w, tex_h;
    const float* sh;
    const float* vnormal;  // [B,C,N,3]
    float* bary;
    int* face;
    float* render;
    int* depth_q;
    int* tie_count;
    bool vec;  // rows of a multiple of four pixels, outputs 16-byte aligned
    // fused image L1 (NULL state: not fused)
    const float* l1_target;
    const unsigned char* l1_mask;
    L1State* l1_state;
};

// colour of a pixel hit by face f at barycentrics (a, bb)
__device__ __forceinline__ float3 shade_pixel(const ShadeArgs& A, const ViewCam& cam, int view, int b, int f,
                                              float a, float bb, float3 dir) {
    const int3 id = A.faces[f];
    // the interpolated normal, only where the albedo or the shading reads it
    float3 pn = make_float3(0.f, 0.f, 0.f);
    if (A.albedo == kNormal || A.albedo == kLighting || A.shading == kShaded) {
        const float* VN = A.vnormal + ((long long)view * A.N) * 3;
        const float3 n0 = ld3(VN + 3 * id.x), n1 = ld3(VN + 3 * id.y), n2 = ld3(VN + 3 * id.z);
        pn = n0 * a + n1 * bb + n2 * (1.f - a - bb);
        pn = pn / length3(pn);
        if (dot(pn, dir) > 0.f) pn = -pn;
    }
    float3 color = make_float3(0.f, 0.f, 0.f);
    switch (A.albedo) {
        case kTextured: {
            const float* tc = A.texcoords + (long long)f * 6;
            const float2 t0 = make_float2(tc[0], 1.f - tc[1]);
            const float2 t1 = make_float2(tc[2], 1.f - tc[3]);
            const float2 t2 = make_float2(tc[4], 1.f - tc[5]);
            float2 uv = t0 * a + t1 * bb + t2 * (1.f - a - bb);
            uv.x = uv.x * A.tex_w;
            uv.y = uv.y * A.tex_h;
            uv.x = fmaxf(uv.x, 0.f);
            uv.x = fminf(uv.x, (float)(A.tex_w - 1));
            uv.y = fmaxf(uv.y, 0.f);
            uv.y = fminf(uv.y, (float)(A.tex_h - 1));
            const int lu = (int)(uv.x - 0.5f);
            const int lv = (int)(uv.y - 0.5f);
            const float* T = A.texture + (long long)b * A.tex_h * A.tex_w * 3;
            color = ld3(T + 3LL * A.tex_w * lv + 3 * lu);
            break;
        }
        case kTexturedBilinear: {
            const float* tc = A.texcoords + (long long)f * 6;
            const float2 t0 = make_float2(tc[0], 1.f - tc[1]);
            const float2 t1 = make_float2(tc[2], 1.f - tc[3]);
            const float2 t2 = make_float2(tc[4], 1.f - tc[5]);
            const float2 uv = t0 * a + t1 * bb + t2 * (1.f - a - bb);
            const float* T = A.texture + (long long)b * A.tex_h * A.tex_w * 3;
            color = bilinear_sample(T, bilinear_taps(uv.x * A.tex_w, uv.y * A.tex_h, A.tex_w, A.tex_h));
            break;
        }
        case kVertexColor: {
            const float* Cc = A.colors + (long long)b * A.N * 3;
            const float3 c0 = ld3(Cc + 3 * id.x), c1 = ld3(Cc + 3 * id.y), c2 = ld3(Cc + 3 * id.z);
            color = make_float3(c0.x * a + c1.x * bb + c2.x * (1.f - a - bb),
                                c0.y * a + c1.y * bb + c2.y * (1.f - a - bb),
                                c0.z * a + c1.z * bb + c2.z * (1.f - a - bb));
            break;
        }
        case kNormal:
            color = make_float3((1.f + pn.x) / 2.f, (1.f + pn.y) / 2.f, (1.f + pn.z) / 2.f);
            break;
        case kLighting:
        case kForegroundMask:
            color = make_float3(1.f, 1.f, 1.f);
            break;
        case kPosition:
        case kDepth: {
            const float* P = A.verts + (long long)b * A.N * 3;
            const float3 p0 = ld3(P + 3 * id.x), p1 = ld3(P + 3 * id.y), p2 = ld3(P + 3 * id.z);
            const float3 pos = make_float3(p0.x * a + p1.x * bb + p2.x * (1.f - a - bb),
                                           p0.y * a + p1.y * bb + p2.y * (1.f - a - bb),
                                           p0.z * a + p1.z * bb + p2.z * (1.f - a - bb));
            if (A.albedo == kPosition) {
                color = pos;
            } else {
                const float3 o = make_float3(cam.ro[0], cam.ro[1], cam.ro[2]);
                const float d = length3(o - pos);
                color = make_float3(d, d, d);
            }
            break;
        }
        case kUV: {
            const float* tc = A.texcoords + (long long)f * 6;
            const float2 t0 = make_float2(tc[0], 1.f - tc[1]);
            const float2 t1 = make_float2(tc[2], 1.f - tc[3]);
            const float2 t2 = make_float2(tc[4], 1.f - tc[5]);
            float2 uv = t0 * a + t1 * bb + t2 * (1.f - a - bb);
            uv.x = fminf(fmaxf(uv.x, 0.f), 1.f);
            uv.y = fminf(fmaxf(uv.y, 0.f), 1.f);
            color = make_float3(uv.x, uv.y, 0.f);
            break;
        }
        default:
            break;
    }
    if ((A.shading == kShaded && A.albedo != kNormal) || A.albedo == kLighting) {
        const float3 L = sh_illum(A.sh + (long long)view * 27, pn);
        color = make_float3(L.x * color.x, L.y * color.y, L.z * color.z);
    }
    return color;
}

// Hit test with an early depth rejection: the quantised depth int(t * 1e4) is
// known as soon as t is, so a triangle that cannot reach the pixel's current
// best depth skips the edge tests; so does a pixel known to lie inside.
// Accepted hits and their depth are those of raster_hit.  The barycentric
// window (a, b <= 1.001 |N|^2 after the sign tests) is decided without the two
// divisions unless a value is near its end or not a number, or |N|^2 is near
// overflow (there the quotients are NaN and the hit is refused); it is never near
// underflow, since |N| is at least the |dir . N| of 1e-7 tested first.
__device__ __forceinline__ bool raster_hit_below(float3 ro_s, float3 dir, const TriS& T, float num,
                                                 unsigned best_d, bool inside, int& depth_q) {
    const float ndr = dot(dir, T.n);
    if (fabsf(ndr) < 0.0000001f) return false;
    const float t = num / ndr;
    if (t < 0.f) return false;
    depth_q = (int)(t * 10000.f);
    if ((unsigned)depth_q > best_d) return false;
    if (inside) return true;
    const float3 P = ro_s + t * dir;
    float3 C = cross(T.s1 - T.s0, P - T.s0);
    if (dot(T.n, C) < 0.f) return false;
    C = cross(T.s2 - T.s1, P - T.s1);
    const float a = dot(T.n, C);
    if (a < 0.f) return false;
    C = cross(T.s0 - T.s2, P - T.s2);
    const float b = dot(T.n, C);
    if (b < 0.f) return false;
    const float denom = dot(T.n, T.n);
    if (denom < 1e30f && a <= 1.0005f * denom && b <= 1.0005f * denom) return true;
    return (a / denom >= -0.001f) && (b / denom >= -0.001f) && (a / denom <= 1.001f) && (b / denom <= 1.001f);
}

__device__ __forceinline__ void store_bary(const ShadeArgs& A, long long pix, float a, float b) {
    if (A.vec) {  // launch-uniform
        reinterpret_cast<float2*>(A.bary)[pix] = make_float2(a, b);
    } else {
        A.bary[2 * pix + 0] = a;
        A.bary[2 * pix + 1] = b;
    }
}

// TIES: the call asked for the per-pixel count of hits at the winning depth
// (diagnostics); without it the count is compiled out, which frees a register
// of the scan and shortens its updates
//
// Resident CTAs claim the tiles of the call (the frame's cameras
// concatenated) from a counter, `claim_n` consecutive tiles per atomic: no
// launch cost per tile, and tiles of very different cost still balance.
//
// A chunk of the tile's bin is copied to shared memory, six consecutive
// threads per 96-byte record, so a warp's copy touches as few lines as the
// records have and passes through no registers (a lane per record takes 32
// lines for each 16-byte piece).  It is then ordered by (back-facing, lower
// bound of the depth within the tile): 32-bit keys (facing | bound | slot) are
// distinct; each warp sorts its 32 keys with a shuffle bitonic network, and a
// key's rank in the chunk is its lane plus its lower bound in every other
// warp's sorted keys (5-step binary searches).
//
// Each warp turns 32 ordered records at a time into per-pixel lists: a lane
// forms the 32-bit mask of the warp's pixels that its triangle can hit
// (pixel_mask), and a bit-matrix transpose hands every pixel the mask of the
// records that can hit it.  A pixel visits only those, nearest bound first,
// front faces before back faces, and leaves a run at the first triangle whose
// bound exceeds its best depth: that one can neither win nor tie, nor can any
// after it in the run.  (Walking all records in lockstep, a pixel visited 19
// and tested 4, and the warp paid every test that one of its pixels needed.)
// The result is the minimum (depth, id) over the triangles whose box holds the
// pixel, as in one unordered pass.
//
// Bound by instruction issue (DRAM at 3-8 % of its rate).  Lists instead of
// the lockstep walk, the bound within the tile instead of the triangle's, and
// claims sized to the call: 16 x 8 views of 1024^2, 8-px tiles 7.50 -> 6.73 ms;
// 2 x 4 mixed-size views of a mesh of long thin triangles 751 -> 496 us;
// 4 x 2048^2 at 16 px 1265 -> 968 us; one 512^2 view 84 -> 20 us.  Whole rows
// of background, copies from a fixed piece per thread, and the image L1 kept
// per thread over all tiles instead of reduced per warp and tile: 6.67 -> 6.05
// ms, 486 -> 418 us, 960 -> 918 us.
template <int TS, bool TIES>
__global__ void __launch_bounds__(TS* TS, TS == 8 ? 20 : (TS == 16 ? 5 : 1)) k_resolve(ShadeArgs A, FastDiv fd_frame,
                                                   const int* __restrict__ tile_cam, int cap,
                                                   const ViewCam* __restrict__ cams,
                                                   const TriFrame* __restrict__ tri_frame,
                                                   const TriView* __restrict__ tri_view,
                                                   const int2* __restrict__ tile_state,
                                                   const int* __restrict__ bins,
                                                   const unsigned long long* __restrict__ spill_keys,
                                                   int spill_tile_cap, long long n_tiles, int claim_n,
                                                   unsigned long long* __restrict__ claim) {
    constexpr int NT = TS * TS;
    constexpr int RW = 32 / TS;                 // pixel rows of a warp
    constexpr int CHUNK = NT > 256 ? 256 : NT;  // triangles staged per round
    constexpr int SB = CHUNK == 64 ? 6 : 8;     // slot bits of a sort key
    constexpr unsigned kNoKey = 0xffffffffu;
    constexpr int kRec = (sizeof(TriView) + sizeof(TriFrame)) / 16;  // 16-byte pieces of a record
    constexpr int kViewRec = sizeof(TriView) / 16;
    static_assert(sizeof(TriView) == 48 && sizeof(TriFrame) == 48, "the copy's stride");
    __shared__ float4 s_rec[CHUNK * kRec];  // staged records (TriView, TriFrame), by slot
    __shared__ unsigned s_key[CHUNK];       // per warp: its keys, sorted
    __shared__ unsigned s_ord[CHUNK];       // the chunk's keys in order
    __shared__ int s_face[CHUNK];           // triangle of each slot
    // thread 0 claims into the slot of this claim's parity; the slot is
    // rewritten two claims later, after every thread has passed the next
    // claim's barrier
    __shared__ long long s_g[2];
    // each thread's share of the image L1 (fused L1 only)
    __shared__ double s_l1[NT];
    __shared__ unsigned s_l1n[NT];
    s_l1[threadIdx.x] = 0.0;
    s_l1n[threadIdx.x] = 0u;
    // the copy of the records: this thread's 16-byte piece and first record
    const int piece = (int)threadIdx.x % kRec, rec0 = (int)threadIdx.x / kRec;
    constexpr int kPerRound = NT / kRec;  // records per round
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned keep = 0;  // bit per stage of the bitonic network: this lane keeps the smaller key
    {
        int at = 0;
#pragma unroll
        for (int size = 2; size <= 32; size <<= 1)
#pragma unroll
            for (int stride = size >> 1; stride > 0; stride >>= 1, ++at)
                keep |= (unsigned)(((lane & stride) == 0) == ((lane & size) == 0)) << at;
    }
    int left = 0, par = 1;  // tiles left of the current claim; its slot
    long long g = 0;
    for (;; --left, ++g) {  // (the background branch continues here too)
    if (left == 0) {
        par ^= 1;
        if (threadIdx.x == 0) s_g[par] = (long long)atomicAdd(claim, (unsigned long long)claim_n);
        __syncthreads();
        g = s_g[par];
        left = claim_n;
    }
    if (g >= n_tiles) break;
    // tile -> (frame, camera, tile of the camera): the call has < 2^31 tiles
    const int b = (int)fd_frame.div((unsigned)g);
    const int view = b * A.C + tile_cam[fd_frame.mod((unsigned)g, (unsigned)b)];
    const ViewCam& cam = cams[view];
    const int tile = (int)(g - cam.tile_base);
    const int W = cam.W, H = cam.H;
    const int ty = (int)cam.fd_tiles_x.div((unsigned)tile), tx = (int)cam.fd_tiles_x.mod((unsigned)tile, ty);
    const int px = tx * TS + threadIdx.x % TS, py = ty * TS + threadIdx.x / TS;
    const float cx = px + 0.5f, cy = py + 0.5f;
    const bool valid = px < W && py < H;
    const int2 st = tile_state[g];
    const int n = min(st.x, cap);
    if (n == 0) {  // background (a tile spills only beyond a full bin)
        const long long pix = cam.pix_base + (long long)py * W + px;
        if (A.vec && (tx + 1) * TS <= W && (ty + 1) * TS <= H) {
            // whole rows: 16-byte stores, TS / 4 of the faces, twice that of the
            // barycentrics, three times of the colours
            constexpr int Q = TS / 4, kStores = TS * 6 * Q;
            const long long first = cam.pix_base + (long long)ty * TS * W + tx * TS;
#pragma unroll
            for (int k = 0; k < (kStores + NT - 1) / NT; ++k) {
                const int i = (int)threadIdx.x + k * NT, row = i / (6 * Q), q = i - row * (6 * Q);
                if (kStores % NT != 0 && i >= kStores) break;
                const long long p = first + (long long)row * W;
                const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
                if (q < 3 * Q) reinterpret_cast<float4*>(A.render + 3 * p)[q] = zero;
                else if (q < 5 * Q) reinterpret_cast<float4*>(A.bary + 2 * p)[q - 3 * Q] = zero;
                else reinterpret_cast<int4*>(A.face + p)[q - 5 * Q] = make_int4(-1, -1, -1, -1);
            }
        } else if (valid) {
            A.face[pix] = -1;
            A.bary[2 * pix + 0] = 0.f;
            A.bary[2 * pix + 1] = 0.f;
            A.render[3 * pix + 0] = 0.f;
            A.render[3 * pix + 1] = 0.f;
            A.render[3 * pix + 2] = 0.f;
        }
        if (valid && A.depth_q) A.depth_q[pix] = 0x7fffffff;
        if (TIES && valid) A.tie_count[pix] = 0;
        continue;
    }
    const float3 ro_s = make_float3(cam.ro_s[0], cam.ro_s[1], cam.ro_s[2]);
    const float3 dir = pixel_ray<true>(cam, px, py);
    const int* tb = bins + g * cap;
    unsigned best_d = 0xffffffffu;
    int best_f = 0x7fffffff;
    int ties = 0;
    int best_e = -1;  // bin entry (base + slot) of the winner, -1 when it came from the spill
    for (int base = 0; base < n; base += CHUNK) {
        const int m = min(CHUNK, n - base);
        __syncthreads();  // the previous chunk's readers are done
        if (rec0 < kPerRound) {
            // both records have kViewRec pieces of a 48-byte stride
            const char* src = piece < kViewRec ? reinterpret_cast<const char*>(tri_view + (long long)view * A.F) + 16 * piece
                                               : reinterpret_cast<const char*>(tri_frame + (long long)b * A.F) + 16 * (piece - kViewRec);
            unsigned dst = (unsigned)__cvta_generic_to_shared(&s_rec[rec0 * kRec + piece]);
            for (int r = rec0; r < m; r += kPerRound, dst += 16 * kRec * kPerRound) {
                const int f = tb[base + r];
                if (piece == 0) s_face[r] = f;
                asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src + 48ll * f));
            }
        }
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncthreads();
        bool front = false;
        unsigned key = kNoKey;
        if ((int)threadIdx.x < m) {
            const float4* rec = s_rec + threadIdx.x * kRec;
            TriFrame tf;
            tf.a = rec[kViewRec];
            tf.b = rec[kViewRec + 1];
            tf.c = rec[kViewRec + 2];
            const float num = rec[2].y;
            const TileRays rays = tile_rays(cam, tx * TS + 0.5f * TS, ty * TS + 0.5f * TS, 0.5f * (TS - 1));
            front = num < 0.f;  // the plane normal points towards the camera
            // the bound, clamped to the key's 31 - SB bits (exact below ~2^25 quanta, a
            // lower bound above) and kept below the all-ones key of an empty slot
            const unsigned coarse = min((unsigned)depth_lower_bound(num, tri_from(tf), ro_s, rays),
                                        (1u << (31 - SB)) - 2u);
            key = (front ? 0u : 0x80000000u) | (coarse << SB) | threadIdx.x;
        }
        if (threadIdx.x < CHUNK && (int)(threadIdx.x & ~31u) < m) {  // whole warps that hold keys
            int at = 0;
#pragma unroll
            for (int size = 2; size <= 32; size <<= 1) {
#pragma unroll
                for (int stride = size >> 1; stride > 0; stride >>= 1, ++at) {
                    const unsigned o = __shfl_xor_sync(0xffffffffu, key, stride);
                    key = (keep >> at) & 1u ? min(key, o) : max(key, o);
                }
            }
            s_key[threadIdx.x] = key;
        }
        const int n_front = __syncthreads_count(front);
        if (threadIdx.x < CHUNK && key != kNoKey) {
            int r = lane;
            const int nw = (m + 31) >> 5;
            for (int w = 0; w < nw; ++w) {
                if (w == warp) continue;
                const unsigned* L = s_key + 32 * w;
                int lo = 0;
#pragma unroll
                for (int step = 16; step > 0; step >>= 1) lo += L[lo + step] < key ? step : 0;
                r += lo + (L[lo] < key ? 1 : 0);
            }
            s_ord[r] = key;
        }
        __syncthreads();
        for (int s0 = 0; s0 < m; s0 += 32) {  // warp-uniform
            const int cnt = min(32, m - s0), nf = min(max(n_front - s0, 0), cnt);  // records, front faces of the group
            // no pixel of the warp can be reached by the group's nearest front or back face
            const unsigned bf = nf > 0 ? s_ord[s0] >> SB : kNoKey;
            const unsigned bb = nf < cnt ? (s_ord[s0 + nf] & 0x7fffffffu) >> SB : kNoKey;
            if (!__any_sync(0xffffffffu, valid && min(bf, bb) <= best_d)) continue;
            unsigned w = 0u;
            if (lane < cnt) {
                const float4* rec = s_rec + (s_ord[s0 + lane] & (CHUNK - 1)) * kRec;
                const float4 ea = rec[0], eb = rec[1], q = rec[2];
                w = pixel_mask<TS, RW>(ea.x, ea.y, eb.z, ea.z, ea.w, eb.w, eb.x, eb.y, q.x, __float_as_int(q.z),
                                       __float_as_int(q.w), tx * TS, ty * TS + warp * RW);
            }
            w = transpose_bits(w, lane);
            if (!valid) w = 0u;
            const unsigned fm = nf == 32 ? 0xffffffffu : (1u << nf) - 1u;  // the front faces' bits
            while (w) {
                const unsigned k = s_ord[s0 + __ffs(w) - 1];
                w &= w - 1u;
                if ((k & 0x7fffffffu) >> SB > best_d) {  // neither this nor a later one of its run can reach the best depth
                    w &= (k >> 31) ? 0u : ~fm;
                    continue;
                }
                const int slot = (int)(k & (CHUNK - 1));
                const float4* rec = s_rec + slot * kRec;
                const float4 ea = rec[0], eb = rec[1], q = rec[2];
                const float e0 = ea.x * cx + ea.y * cy + eb.z, e1 = ea.z * cx + ea.w * cy + eb.w,
                            e2 = eb.x * cx + eb.y * cy + q.x;
                if (e0 < 0.f || e1 < 0.f || e2 < 0.f) continue;  // clearly outside the projected triangle
                TriFrame tf;
                tf.a = rec[kViewRec];
                tf.b = rec[kViewRec + 1];
                tf.c = rec[kViewRec + 2];
                // clearly inside: the edge tests would pass, only the depth is needed
                const bool inside = e0 >= kEdgeInterior && e1 >= kEdgeInterior && e2 >= kEdgeInterior;
                int dq;
                if (!raster_hit_below(ro_s, dir, tri_from(tf), q.y, best_d, inside, dq)) continue;
                const int f = s_face[slot];
                if ((unsigned)dq < best_d) {
                    best_d = (unsigned)dq;
                    best_f = f;
                    best_e = base + slot;
                    ties = 1;
                } else {  // equal depth (deeper hits were rejected)
                    if (f < best_f) {
                        best_f = f;
                        best_e = base + slot;
                    }
                    ++ties;
                }
            }
        }
    }
    if (valid) {
        if (st.x > cap && st.y > 0 && st.y <= spill_tile_cap) {
            const unsigned long long key = spill_keys[(long long)(st.y - 1) * NT + threadIdx.x];
            if (key != ~0ull) {
                const unsigned kd = (unsigned)(key >> 32);
                const int kf = (int)(key & 0xffffffffu);
                if (kd < best_d) {
                    best_d = kd;
                    best_f = kf;
                    best_e = -1;
                    ties = 0;  // spilled ties are added by the diagnostics pass
                } else if (kd == best_d && kf < best_f) {
                    best_f = kf;
                    best_e = -1;
                }
            }
        }
        const long long pix = cam.pix_base + (long long)py * W + px;
        if (best_d == 0xffffffffu) {
            A.face[pix] = -1;
            store_bary(A, pix, 0.f, 0.f);
            A.render[3 * pix + 0] = 0.f;
            A.render[3 * pix + 1] = 0.f;
            A.render[3 * pix + 2] = 0.f;
            if (A.depth_q) A.depth_q[pix] = 0x7fffffff;
            if (TIES) A.tie_count[pix] = 0;
        } else {
            // the fused L1's target, loaded before this pixel's stores (which
            // the compiler may not move it past)
            const bool l1m = A.l1_state && (!A.l1_mask || A.l1_mask[pix]);
            const float3 tg = l1m ? ld3(A.l1_target + 3 * pix) : make_float3(0.f, 0.f, 0.f);
            // recompute the winner's barycentrics (same arithmetic as the hit test)
            // the winner's triangle and plane offset: from the staged chunk when
            // the winner is in the last one staged (s_rec is rewritten only
            // after the next tile's first barrier), else from global memory
            const int last_base = n > 0 ? ((n - 1) / CHUNK) * CHUNK : 0;
            TriS Tw;
            float wnum;
            if (best_e >= last_base) {
                const float4* rec = s_rec + (best_e - last_base) * kRec;
                TriFrame tf;
                tf.a = rec[kViewRec];
                tf.b = rec[kViewRec + 1];
                tf.c = rec[kViewRec + 2];
                Tw = tri_from(tf);
                wnum = rec[2].y;
            } else {
                Tw = tri_from(tri_frame[(long long)b * A.F + best_f]);
                wnum = tri_view[(long long)view * A.F + best_f].num;
            }
            float a, bb;
            winner_bary(ro_s, dir, Tw, wnum, a, bb);
            // every load of the shading before the first store of the pixel
            const float3 col = shade_pixel(A, cam, view, b, best_f, a, bb, dir);
            A.face[pix] = best_f;
            store_bary(A, pix, a, bb);
            A.render[3 * pix + 0] = col.x;
            A.render[3 * pix + 1] = col.y;
            A.render[3 * pix + 2] = col.z;
            if (A.depth_q) A.depth_q[pix] = (int)best_d;
            if (TIES) A.tie_count[pix] = ties;
            if (l1m) {
                const float d0 = l1_diff(col.x, tg.x), d1 = l1_diff(col.y, tg.y), d2 = l1_diff(col.z, tg.z);
                s_l1[threadIdx.x] += (double)(fabsf(d0) + fabsf(d1) + fabsf(d2));
                s_l1n[threadIdx.x] += (d0 != 0.f) + (d1 != 0.f) + (d2 != 0.f);
            }
        }
    }
    }
    if (A.l1_state) {  // launch-uniform: the CTA's image L1, one atomic pair per warp
        double l1s = s_l1[threadIdx.x];
        unsigned long long l1c = s_l1n[threadIdx.x];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            l1s += __shfl_xor_sync(0xffffffffu, l1s, o);
            l1c += __shfl_xor_sync(0xffffffffu, l1c, o);
        }
        if (lane == 0 && l1c) {
            atomicAdd(&A.l1_state->sum, l1s);
            atomicAdd(&A.l1_state->count, l1c);
        }
    }
}

__global__ void k_l1_loss(const L1State* __restrict__ state, float* __restrict__ loss) {
    const unsigned long long c = state->count;
    *loss = c ? (float)(state->sum / (double)c) : 0.f;
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
// Tiles a CTA of the tile resolve claims per atomic: four, so that the one
// counter sees a quarter of the atomics, but no more than leave every CTA at
// least four claims (a 512 x 512 view has 1024 tiles of 16 px for 740 CTAs:
// claims of four would leave two thirds of them idle)
static int claim_size(long long tiles, unsigned grid) {
    return (int)std::max<long long>(1, std::min<long long>(4, tiles / (4ll * grid)));
}

// Per-camera layout of a frame for the current tile size: each camera's
// resolution, tile grids and offsets, and the camera of every tile (the tile
// resolve and the adjoint launch one CTA per tile of the whole call).
hc_status raster_layout(RasterWorkspace& ws) {
    const int TS = ws.tile, C = (int)ws.cam_w.size();
    if (ws.layout_tile == TS) return HC_OK;
    std::vector<CamLayout> L(C);
    std::vector<int> tc, tcb;
    long long pix = 0, tile = 0, tile_b = 0;
    for (int c = 0; c < C; ++c) {
        CamLayout& l = L[c];
        l.W = ws.cam_w[c];
        l.H = ws.cam_h[c];
        l.tiles_x = div_up(l.W, TS);
        l.tiles_x_b = div_up(l.W, kAdjointTile);
        l.fd_tiles_x = FastDiv((unsigned)l.tiles_x);
        l.fd_tiles_x_b = FastDiv((unsigned)l.tiles_x_b);
        l.pix = pix;
        l.tile = tile;
        l.tile_b = tile_b;
        const long long nt = (long long)l.tiles_x * div_up(l.H, TS);
        const long long ntb = (long long)l.tiles_x_b * div_up(l.H, kAdjointTile);
        tc.insert(tc.end(), (size_t)nt, c);
        tcb.insert(tcb.end(), (size_t)ntb, c);
        pix += (long long)l.W * l.H;
        tile += nt;
        tile_b += ntb;
    }
    HC_TRY(upload(ws.layout, L.data(), L.size()));
    HC_TRY(upload(ws.tile_cam, tc.data(), tc.size()));
    HC_TRY(upload(ws.tile_cam_b, tcb.data(), tcb.size()));
    ws.P_frame = pix;
    ws.T_frame = tile;
    ws.Tb_frame = tile_b;
    ws.layout_tile = TS;
    ws.cap_views = 0;  // bins depend on the tile count
    return HC_OK;
}

hc_status raster_reserve(RasterWorkspace& ws, int views, int F) {
    HC_TRY(raster_layout(ws));
    const int TS = ws.tile;
    const int C = (int)ws.cam_w.size();
    const long long tiles = (long long)(views / C) * ws.T_frame;  // all tiles of the call
    if (views > ws.cap_views || ws.bins.bytes < (size_t)tiles * ws.bin_cap * sizeof(int)) {
        HC_TRY(ws.cams.ensure(sizeof(ViewCam) * views));
        if (ws.vacc_floats && ws.size_vacc() != HC_OK) {  // an adjoint that needs it will say so
            clear_error();
        }
        HC_TRY(ws.tri_view.ensure(sizeof(TriView) * (size_t)views * F));
        HC_TRY(ws.tile_state.ensure(sizeof(int2) * (size_t)tiles));
        HC_TRY(ws.bins.ensure(sizeof(int) * (size_t)tiles * ws.bin_cap));
        // crumpled meshes overflow many bins: room for four spilled pairs per
        // (view, triangle), and a key block for every tile while that stays
        // under 4 GB (a quarter of the tiles beyond); overflow is reported by
        // hc_renderer_stats
        ws.spill_cap = std::max<long long>(1 << 22, 4ll * views * F);
        HC_TRY(ws.spill.ensure(sizeof(int2) * (size_t)ws.spill_cap));
        const long long per_tile = (long long)TS * TS * sizeof(unsigned long long);
        ws.spill_tile_cap = (int)(tiles * per_tile <= (4ll << 30) ? tiles : std::max<long long>(256, tiles / 4));
        HC_TRY(ws.spill_keys.ensure(sizeof(unsigned long long) * (size_t)ws.spill_tile_cap * TS * TS));
        HC_TRY(ws.stats.ensure(sizeof(RasterStats)));
        HC_TRY(ws.claim.ensure(sizeof(unsigned long long)));
        HC_TRY(ws.claim_b.ensure(sizeof(unsigned)));
        ws.cap_views = views;
    }
    return HC_OK;
}

hc_status raster_forward(const Topology& topo, RasterWorkspace& ws, cudaStream_t s, int B, int C, int albedo,
                         int shading, const float* verts, const float* colors, const float* texture, int tex_h,
                         int tex_w, const float* sh, const float* extr, const float* intr, float* bary, int* face,
                         float* render, float* vnormal, int* depth_q, int* tie_count, const L1Fuse* l1) {
    const int V = B * C;
    const int N = topo.N, F = topo.F;
    HC_TRY(raster_reserve(ws, V, F));
    HC_TRY(ws.tri_frame.ensure(sizeof(TriFrame) * (size_t)B * F));
    HC_TRY(ws.proj.ensure(sizeof(float4) * (size_t)V * N));
    const int TS = ws.tile;
    const long long tiles = (long long)B * ws.T_frame;
    ViewCam* cams = ws.cams.as<ViewCam>();
    TriFrame* tf = ws.tri_frame.as<TriFrame>();
    TriView* tv = ws.tri_view.as<TriView>();
    int2* tstate = ws.tile_state.as<int2>();
    RasterStats* stats = ws.stats.as<RasterStats>();

    unsigned long long* claim = ws.claim.as<unsigned long long>();

    FillRuns zeros;
    zeros.add(tstate, sizeof(int2) * (size_t)tiles);
    zeros.add(stats, sizeof(RasterStats));
    zeros.add(claim, sizeof(unsigned long long));
    if (l1) zeros.add(l1->state, sizeof(L1State));
    const int view_blocks = div_up(V, kViewThreads);
    ws.clock.begin(kKViewSetup, s);
    k_view_setup<<<view_blocks + zeros.blocks(kViewThreads), kViewThreads, 0, s>>>(
        V, C, extr, intr, ws.layout.as<CamLayout>(), ws.P_frame, ws.T_frame, ws.Tb_frame, cams, view_blocks, zeros);
    HC_CHECK_LAUNCH();
    ws.clock.end(kKViewSetup, s);
    FrameSetup S;
    S.B = B;
    S.C = C;
    S.N = N;
    S.F = F;
    S.faces = topo.faces.as<int3>();
    S.fan = topo.fan.as<int2>();
    S.vf_id = topo.vf_id.as<int2>();
    S.verts = verts;
    S.vnormal = vnormal;
    S.unit = nullptr;
    S.tri = tf;
    S.cams = cams;
    S.proj = ws.proj.as<float4>();
    // kernel timing names the parts: a launch each then
    const unsigned nb = div_up((long long)B * N, kSetupThreads), fb = div_up((long long)B * F, kSetupThreads),
                   pb = div_up((long long)V * N, kSetupThreads);
    auto setup = [&](unsigned normals, unsigned tris, unsigned projected) -> hc_status {
        S.normal_blocks = normals;
        S.tri_blocks = tris;
        S.project_blocks = projected;
        k_frame_setup<<<normals + tris + projected, kSetupThreads, 0, s>>>(S);
        HC_CHECK_LAUNCH();
        return HC_OK;
    };
    if (ws.clock.on) {
        ws.clock.begin(kKVertexNormals, s);
        HC_TRY(setup(nb, 0, 0));
        ws.clock.end(kKVertexNormals, s);
        ws.clock.begin(kKTriFrame, s);
        HC_TRY(setup(0, fb, 0));
        ws.clock.end(kKTriFrame, s);
        ws.clock.begin(kKBin, s);
        HC_TRY(setup(0, 0, pb));
    } else {
        HC_TRY(setup(nb, fb, pb));
    }
    HC_REQUIRE(V <= 65535, "too many views in one call (%d)", V);
    HC_REQUIRE(tiles < (1ll << 31), "too many tiles in one call (%lld)", tiles);
    const int ts_shift = TS == 8 ? 3 : (TS == 16 ? 4 : 5);
    HC_REQUIRE(TS == (1 << ts_shift), "tile size %d is not 8, 16 or 32", TS);
    k_bin<<<dim3(div_up(F, 256), V), 256, 0, s>>>(
        V, C, F, N, TS, ts_shift, ws.bin_cap, topo.faces.as<int3>(), ws.proj.as<float4>(), cams, tf, tv, tstate,
        ws.bins.as<int>(),
        ws.spill.as<int2>(), ws.spill_cap, ws.spill_keys.as<unsigned long long>(), ws.spill_tile_cap, stats);
    HC_CHECK_LAUNCH();
    ws.clock.end(kKBin, s);
    ws.clock.begin(kKSpill, s);
    k_spill<<<148 * 4, 128, 0, s>>>(C, F, TS, ws.T_frame, ws.tile_cam.as<int>(), cams, tf, tv, tstate,
                                    ws.spill.as<int2>(), ws.spill_cap,
                                    ws.spill_tile_cap, ws.spill_keys.as<unsigned long long>(), stats, nullptr,
                                    nullptr);
    HC_CHECK_LAUNCH();
    ws.clock.end(kKSpill, s);
    ShadeArgs A;
    A.B = B;
    A.C = C;
    A.N = N;
    A.F = F;
    A.albedo = albedo;
    A.shading = shading;
    A.faces = topo.faces.as<int3>();
    A.texcoords = topo.texcoords.as<float>();
    A.verts = verts;
    A.colors = colors;
    A.texture = texture;
    A.tex_w = tex_w;
    A.tex_h = tex_h;
    A.sh = sh;
    A.vnormal = vnormal;
    A.bary = bary;
    A.face = face;
    A.render = render;
    A.depth_q = depth_q;
    A.tie_count = tie_count;
    A.vec = (((uintptr_t)bary | (uintptr_t)face | (uintptr_t)render) & 15) == 0;
    for (int w : ws.cam_w) A.vec = A.vec && w % 4 == 0;
    A.l1_target = l1 ? l1->target : nullptr;
    A.l1_mask = l1 ? l1->mask : nullptr;
    A.l1_state = l1 ? l1->state : nullptr;
    const int* tcam = ws.tile_cam.as<int>();
    HC_REQUIRE(tiles < (1ll << 31), "too many tiles in one call (%lld)", tiles);
    const int* kbins = ws.bins.as<int>();
    const unsigned long long* kspill = ws.spill_keys.as<unsigned long long>();
    ws.clock.begin(kKResolve, s);
#define HC_RESOLVE_CASE(TSV)                                                                                   \
    case TSV: {                                                                                                \
        auto kernel = A.tie_count ? k_resolve<TSV, true> : k_resolve<TSV, false>;                              \
        const unsigned grid = resident_grid(kernel, TSV * TSV, tiles);                                         \
        kernel<<<grid, TSV * TSV, 0, s>>>(A, FastDiv((unsigned)ws.T_frame), tcam, ws.bin_cap, cams, tf, tv, tstate, \
                                          kbins, kspill, ws.spill_tile_cap, tiles,                             \
                                          claim_size(tiles, grid), claim);                                     \
        break;                                                                                                 \
    }
    switch (TS) {
        HC_RESOLVE_CASE(8)
        HC_RESOLVE_CASE(16)
        HC_RESOLVE_CASE(32)
        default:
            HC_FAIL(HC_ERR_INVALID, "unsupported tile size %d", TS);
    }
#undef HC_RESOLVE_CASE
    HC_CHECK_LAUNCH();
    ws.clock.end(kKResolve, s);
    if (l1) {
        if (l1->loss) {
            k_l1_loss<<<1, 1, 0, s>>>(l1->state, l1->loss);
            HC_CHECK_LAUNCH();
        }
    }
    if (tie_count && depth_q) {
        k_spill<<<148 * 4, 128, 0, s>>>(C, F, TS, ws.T_frame, ws.tile_cam.as<int>(), cams, tf, tv, tstate,
                                    ws.spill.as<int2>(), ws.spill_cap,
                                        ws.spill_tile_cap, ws.spill_keys.as<unsigned long long>(), stats, depth_q,
                                        tie_count);
        HC_CHECK_LAUNCH();
    }
    return HC_OK;
}

}  // namespace hc
