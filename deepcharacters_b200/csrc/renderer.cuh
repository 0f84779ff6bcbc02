// Shared state and device helpers of the rasterizer (forward and adjoint).
//
// Layout in HBM (V = B*C views, T = tiles per view):
//   ViewCam   cams[V]             camera set-up, one per view
//   TriFrame  tri_frame[B*F]      per-frame triangle constants (scaled vertices, plane normal)
//   TriView   tri_view[V*F]       per-view triangle constants (footprint, ray-plane numerator, pixel bbox)
//   int2      tile_state[V*T]     (binned count, spill slot + 1)
//   int       bins[V*T*CAP]       triangle ids per tile
//   int4      spill[S]            (view, tile, triangle) pairs beyond CAP
//   u64       spill_keys[K*TS*TS] packed (depth_q << 32 | triangle) per spilled tile pixel
#pragma once

#include <vector>

#include "hc_common.cuh"
#include "hc_math.cuh"

namespace hc {

enum AlbedoMode {
    kVertexColor = 0, kTextured, kNormal, kLighting, kForegroundMask, kPosition, kDepth, kUV,
    // bilinear texture sampling (no reference counterpart: the reference's
    // textured mode samples the nearest texel, CUDABasedRasterization.cu:347-373)
    kTexturedBilinear
};
enum ShadingMode { kShaded = 0, kShadeless };
enum NormalMapMode { kNmOriginal = 0, kNmHitPosition, kNmNone, kNmFace };

struct ViewCam {
    float invP[16];  // inverse(K * E), row-major 4x4
    float invE[16];  // inverse(E)
    float ext[12];   // world -> camera, row-major 3x4
    float intr[9];   // row-major 3x3
    float ro[3];     // ray origin (camera centre)
    float ro_s[3];   // ray origin / 1000
    float KE[9];     // K * E[:, :3] (row-major): world -> homogeneous pixel, linear part
    float Kt[3];     // K * E[:, 3]
    // the view's image: resolution, tile grids and where its pixels / tiles
    // start in the call's buffers (cameras of a frame may differ in size)
    int W, H, tiles_x, tiles_x_b;
    long long pix_base, tile_base, tile_base_b;
    FastDiv fd_tiles_x, fd_tiles_x_b;  // division by tiles_x / tiles_x_b
};

constexpr int kAdjointTile = 16;  // tile edge of the renderer adjoint

// Values that the adjoint sums per vertex (position; colour with vertex colours;
// normal if shaded), and the floats they take: a multiple of 16 bytes.
__host__ __device__ constexpr int vertex_sum_values(bool vertex_colors, bool shaded) {
    return 3 + (vertex_colors ? 3 : 0) + (shaded ? 3 : 0);
}
__host__ __device__ constexpr int vertex_sum_floats(bool vertex_colors, bool shaded) {
    return (vertex_sum_values(vertex_colors, shaded) + 3) / 4 * 4;
}

// One camera's image inside a frame: the frame's cameras are concatenated,
// so views of different resolutions share one launch.
struct CamLayout {
    int W, H;
    int tiles_x, tiles_x_b;        // raster tiles (ws.tile px) / adjoint tiles (16 px) per row
    long long pix, tile, tile_b;   // first pixel / raster tile / adjoint tile in the frame
    FastDiv fd_tiles_x, fd_tiles_x_b;
};

struct TriFrame {    // 48 bytes: s0.xyz n.x | s1.xyz n.y | s2.xyz n.z
    float4 a, b, c;
};

struct __align__(16) TriView {  // 48 bytes per (view, triangle), written by the binning pass
    float4 e01;      // 2-D footprint edges 0 and 1: (a0, b0, a1, b1)
    float4 e2c;      // edge 2 and two offsets: (a2, b2, c0, c1)
    float c2;        // the third offset
    float num;       // dot(s0, n) - dot(ro_s, n)
    int x01;         // bbox x0 | x1 << 16
    int y01;         // bbox y0 | y1 << 16
};

struct TriS;


struct RasterStats {
    unsigned long long binned;
    unsigned long long spilled;
    int spill_tiles;
    int overflow;      // bit 0: spill list full, bit 1: spill tile slots exhausted,
                       // bit 2: an adjoint target copy (TMA) did not complete
};

// Pixel-centre camera ray (reference getRayCuda2 / backprojectPixelCuda,
// CudaRenderer/cpp/src/Utils/CameraUtil.h:223-258): the pixel centre is lifted
// to depth 1000 through inv(K*E) and the direction from the camera centre is
// normalised with rsqrtf.  The roundings are written out: left to the compiler,
// the order in which it contracts a row's products changes with the code
// around it, and with it the last bits of a ray and the side of an edge that it
// falls on.  In the tile resolve (RESOLVE) the x row rounds its first product
// before the second is added, elsewhere its second, as the other rows do.
template <bool FIRST>
__device__ __forceinline__ float lifted(const float* m, float u, float v) {
    const float s = FIRST ? __fmaf_rn(m[1], v, __fmul_rn(m[0], u)) : __fmaf_rn(m[0], u, __fmul_rn(m[1], v));
    return __fadd_rn(__fmaf_rn(m[2], 1000.f, s), m[3]);
}

template <bool RESOLVE>
__device__ __forceinline__ float3 pixel_ray(const ViewCam& c, int px, int py) {
    const float u = __fmul_rn(px + 0.5f, 1000.f), v = __fmul_rn(py + 0.5f, 1000.f);
    const float3 q = make_float3(lifted<RESOLVE>(c.invP, u, v), lifted<false>(c.invP + 4, u, v),
                                 lifted<false>(c.invP + 8, u, v));
    const float3 d = q - make_float3(c.ro[0], c.ro[1], c.ro[2]);
    return d * rsqrtf(__fmaf_rn(d.z, d.z, __fmaf_rn(d.x, d.x, __fmul_rn(d.y, d.y))));
}

struct TriS {
    float3 s0, s1, s2, n;
};

__device__ __forceinline__ TriS tri_from(const TriFrame& f) {
    TriS t;
    t.s0 = make_float3(f.a.x, f.a.y, f.a.z);
    t.s1 = make_float3(f.b.x, f.b.y, f.b.z);
    t.s2 = make_float3(f.c.x, f.c.y, f.c.z);
    t.n = make_float3(f.a.w, f.b.w, f.c.w);
    return t;
}

// The unnormalised camera rays of a tile's pixel centres: u(x, y) = c + x ux +
// y uy for |x|, |y| <= h pixels from the tile's centre (pixel_ray's affine
// form before its normalisation).  min_len bounds |u| from below; slack
// bounds the float error of u . n over |n|.
struct TileRays {
    float3 c, ux, uy;  // ux, uy scaled by h
    float min_len, slack;
};

__device__ __forceinline__ TileRays tile_rays(const ViewCam& cam, float x, float y, float h) {
    const float* m = cam.invP;
    TileRays r;
    const float3 o = make_float3(cam.ro[0], cam.ro[1], cam.ro[2]);
    r.c = make_float3(1000.f * (m[0] * x + m[1] * y + m[2]) + m[3] - o.x,
                      1000.f * (m[4] * x + m[5] * y + m[6]) + m[7] - o.y,
                      1000.f * (m[8] * x + m[9] * y + m[10]) + m[11] - o.z);
    const float k = 1000.f * h;
    r.ux = make_float3(k * m[0], k * m[4], k * m[8]);
    r.uy = make_float3(k * m[1], k * m[5], k * m[9]);
    const float len = sqrtf(dot(r.c, r.c)), far = fabsf(o.x) + fabsf(o.y) + fabsf(o.z);
    r.slack = 2e-6f * (len + far);
    r.min_len = fmaxf(len - sqrtf(dot(r.ux, r.ux)) - sqrtf(dot(r.uy, r.uy)) - r.slack, 0.f);
    return r;
}

// Conservative lower bound of int(t * 1e4) of a triangle's hits in a tile.
// For the unit ray direction u / |u|, t is the distance from the camera
// centre to the hit point.  It is (a) on the triangle's plane, t = num |u| /
// (u . n), so at least |num| min |u| / max |u . n|, the maximum of the affine
// u . n over the tile being |c . n| + |ux . n| + |uy . n|; and (b) at least the
// distance to the nearest vertex minus the longest edge (every point of a
// triangle lies within its longest edge of some vertex).  The larger of the
// two is lowered by 1e-4 relative and 2 quanta so float rounding of either
// side cannot break it.  (a) is nearly the triangle's depth in the tile: the
// bound of the whole triangle that it replaced left long thin triangles, whose
// nearest point lies far outside the tile, at the head of many tiles.
__device__ __forceinline__ int depth_lower_bound(float num, const TriS& T, float3 o, const TileRays& r) {
    const float most = fabsf(dot(r.c, T.n)) + fabsf(dot(r.ux, T.n)) + fabsf(dot(r.uy, T.n)) +
                       r.slack * (fabsf(T.n.x) + fabsf(T.n.y) + fabsf(T.n.z));
    const float pd = most > 0.f ? fabsf(num) * r.min_len / most : 0.f;
    const float3 a0 = T.s0 - o, a1 = T.s1 - o, a2 = T.s2 - o;
    const float dmin = sqrtf(fminf(dot(a0, a0), fminf(dot(a1, a1), dot(a2, a2))));
    const float3 e0 = T.s1 - T.s0, e1 = T.s2 - T.s1, e2 = T.s0 - T.s2;
    const float e = sqrtf(fmaxf(dot(e0, e0), fmaxf(dot(e1, e1), dot(e2, e2))));
    const float vd = dmin - e;
    const float z = fmaxf(pd, vd) * 10000.f * (1.f - 1e-4f);
    if (!(z < 2.0e9f)) return 0x7fffffff;
    return max((int)z - 2, 0);
}

// Ray / triangle test of the reference (rayTriangleIntersect,
// CudaRenderer/cpp/src/Utils/RendererUtil.h:26-101) with the per-triangle and
// per-view terms hoisted: s* = vertices / 1000, n = cross(s1 - s0, s2 - s0),
// num = dot(s0, n) - dot(origin / 1000, n).  Same operations in the same order
// per pixel, so hit decisions, t and the barycentrics (a weights s0, b weights
// s1) match the reference bit for bit.
__device__ __forceinline__ bool ray_tri(float3 ro_s, float3 dir, const TriS& T, float num,
                                        float& t, float& a, float& b) {
    const float ndr = dot(dir, T.n);
    if (fabsf(ndr) < 0.0000001f) return false;
    t = num / ndr;
    if (t < 0.f) return false;
    const float3 P = ro_s + t * dir;
    float3 C = cross(T.s1 - T.s0, P - T.s0);
    if (dot(T.n, C) < 0.f) return false;
    C = cross(T.s2 - T.s1, P - T.s1);
    if ((a = dot(T.n, C)) < 0.f) return false;
    C = cross(T.s0 - T.s2, P - T.s2);
    if ((b = dot(T.n, C)) < 0.f) return false;
    const float denom = dot(T.n, T.n);
    a /= denom;
    b /= denom;
    return true;
}

// Barycentrics of a pixel's known winner: the operations of ray_tri that
// form a and b, without the sign and window checks that the winner has
// passed (so the values are ray_tri's).
__device__ __forceinline__ void winner_bary(float3 ro_s, float3 dir, const TriS& T, float num, float& a, float& b) {
    const float ndr = dot(dir, T.n);
    const float t = num / ndr;
    const float3 P = ro_s + t * dir;
    float3 C = cross(T.s2 - T.s1, P - T.s1);
    a = dot(T.n, C);
    C = cross(T.s0 - T.s2, P - T.s2);
    b = dot(T.n, C);
    const float denom = dot(T.n, T.n);
    a /= denom;
    b /= denom;
}

// Hit accepted by the depth pass: barycentric window of
// CUDABasedRasterization.cu:243 and the quantised depth int(t * 1e4) of :247-250.
__device__ __forceinline__ bool raster_hit(float3 ro_s, float3 dir, const TriS& T, float num,
                                           int& depth_q, float& a, float& b) {
    float t;
    if (!ray_tri(ro_s, dir, T, num, t, a, b)) return false;
    if (!((a >= -0.001f) && (b >= -0.001f) && (a <= 1.001f) && (b <= 1.001f))) return false;
    depth_q = (int)(t * 10000.f);
    return true;
}

// World -> camera -> pixel projection (reference getCamSpacePoint and
// projectPointFloat3, CudaRenderer/cpp/src/Utils/CameraUtil.h:141-186).
__device__ __forceinline__ float3 project_point(const float* ext, const float* intr, float3 p) {
    const float4 h = make_float4(p.x, p.y, p.z, 1.f);
    const float3 cs = make_float3(dot(make_float4(ext[0], ext[1], ext[2], ext[3]), h),
                                  dot(make_float4(ext[4], ext[5], ext[6], ext[7]), h),
                                  dot(make_float4(ext[8], ext[9], ext[10], ext[11]), h));
    const float3 d1 = cs * make_float3(intr[0], intr[1], intr[2]);
    const float3 d2 = cs * make_float3(intr[3], intr[4], intr[5]);
    const float3 d3 = cs * make_float3(intr[6], intr[7], intr[8]);
    float x = d1.x + d1.y + d1.z;
    float y = d2.x + d2.y + d2.z;
    float z = d3.x + d3.y + d3.z;
    if (z > 0.0000001f) {
        x /= z;
        y /= z;
    } else {
        z = 0.00001f;
        x /= z;
        y /= z;
    }
    return make_float3(x, y, z);
}

// Conservative 2-D footprint of a triangle in a view: the three edge lines of
// its projection, each widened by a margin, as signed pixel distances that
// are non-negative inside.  A pixel centre outside the widened triangle
// cannot pass the exact test that follows:
//  * the ray test: for vertices in front of the camera the projected
//    triangle is the exact image of the 3-D one, and the float error of
//    either computation is below 1e-3 px for the coordinate ranges admitted
//    here (|u|, |v| < 1e5 px, z > 1), against a margin of kEdgeMargin px;
//  * the image-space barycentric test with its -0.001 tolerance: edge k is
//    additionally widened by 0.0011 x the triangle's height over that edge,
//    and by num_err / |edge k| px, num_err bounding the rounding error of
//    that test's edge-function numerator (2e-6 M^2 for coordinates up to M).
// Outside that coordinate range, or for a projected area under 1e-2 px^2, the
// footprint is disabled (every pixel passes).  It only skips work; it never
// decides a hit.
constexpr float kEdgeMargin = 0.125f;

struct Footprint {
    float a[3], b[3], c[3];  // edge k: a*x + b*y + c >= 0 inside (margin included)
    float m[3];              // the margin folded into c[k] (0 when disabled)
};
// A pixel centre whose three footprint values are all >= kEdgeInterior lies
// inside the (unwidened) projected triangle by more than kEdgeMargin px: the
// exact ray test's edge and barycentric-window checks certainly pass there.
// (A disabled footprint has values 0 and never qualifies.)
constexpr float kEdgeInterior = 2.f * kEdgeMargin;

__device__ __forceinline__ Footprint footprint(float3 p0, float3 p1, float3 p2, float rel_margin = 0.f,
                                               float num_err = 0.f) {
    Footprint fp;
    const float3 q[3] = {p0, p1, p2};
    bool ok = p0.z > 1.f && p1.z > 1.f && p2.z > 1.f;
#pragma unroll
    for (int k = 0; k < 3; ++k) ok = ok && fabsf(q[k].x) < 1e5f && fabsf(q[k].y) < 1e5f;
    const float area = (p1.x - p0.x) * (p2.y - p0.y) - (p1.y - p0.y) * (p2.x - p0.x);
    ok = ok && fabsf(area) >= 1e-2f;
    const float sg = area > 0.f ? 1.f : -1.f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float3 u = q[k], w = q[(k + 1) % 3];
        const float ex = w.x - u.x, ey = w.y - u.y;
        const float len = sqrtf(ex * ex + ey * ey);
        if (!(len > 1e-6f)) ok = false;
        const float inv = ok ? sg / len : 0.f;
        // (the widenings are skipped when both are zero: 0 / len is not
        // folded away by the compiler, and adds nothing)
        const bool widen = ok && (rel_margin != 0.f || num_err != 0.f);
        const float margin = kEdgeMargin + (widen ? rel_margin * fabsf(area) / len + num_err / len : 0.f);
        // signed distance of (x, y) from the edge u -> w, positive on the inside
        fp.a[k] = -ey * inv;
        fp.b[k] = ex * inv;
        fp.c[k] = (ey * u.x - ex * u.y) * inv + margin;
        fp.m[k] = ok ? margin : 0.f;
    }
    if (!ok) {  // disabled: every pixel is on the boundary band (passes, never "inside")
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            fp.a[k] = 0.f;
            fp.b[k] = 0.f;
            fp.c[k] = 0.f;
            fp.m[k] = 0.f;
        }
    }
    return fp;
}

// false when no pixel centre of [x0, x1] x [y0, y1] can be inside the footprint
__device__ __forceinline__ bool footprint_overlaps(const Footprint& fp, int x0, int x1, int y0, int y1) {
    const float xa = x0 + 0.5f, xb = x1 + 0.5f, ya = y0 + 0.5f, yb = y1 + 0.5f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float m = fp.a[k] * (fp.a[k] > 0.f ? xb : xa) + fp.b[k] * (fp.b[k] > 0.f ? yb : ya) + fp.c[k];
        if (m < 0.f) return false;
    }
    return true;
}

// The same for the rows of a box, an interval of columns per row: edge k leaves
// or enters a row [y0, y1] at x = s y + c for the better of its ends.  A pixel
// column outside the interval fails one edge in every pixel of the row.  Against
// a test of each tile of the box it costs one row's share of the edges, and no
// tile that is missed is visited.  (Each value differs from the sum above by
// rounding only, at most 0.05 px of the edge's distance against its margin of
// kEdgeMargin; edges with a nearly 0 bound no column.)
struct TileRows {
    float s[3], c[3];
    int low;  // bit k: edge k bounds the columns from below; bit 3 + k: b > 0
    __device__ __forceinline__ TileRows() {}
    __device__ __forceinline__ explicit TileRows(const Footprint& fp) : low(0) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const bool bounds = fabsf(fp.a[k]) > 1e-6f;
            const float inv = __fdividef(-1.f, fp.a[k]);
            s[k] = bounds ? fp.b[k] * inv : 0.f;
            c[k] = bounds ? fp.c[k] * inv - 0.5f : -1e30f;
            low |= (!bounds || fp.a[k] > 0.f ? 1 << k : 0) | (fp.b[k] > 0.f ? 8 << k : 0);
        }
    }
    // pixel columns of the row inside [x0, x1]; none if hi < lo
    __device__ __forceinline__ void span(int x0, int x1, int y0, int y1, int& lo, int& hi) const {
        const float ya = y0 + 0.5f, yb = y1 + 0.5f;
        float l = (float)x0, h = (float)x1;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float x = s[k] * (low & (8 << k) ? yb : ya) + c[k];
            if (low & (1 << k)) l = fmaxf(l, x);
            else h = fminf(h, x);
        }
        lo = __float2int_ru(fminf(l, x1 + 1.f));
        hi = __float2int_rd(fmaxf(h, x0 - 1.f));
    }
    // the tiles (edge 1 << sh) of a box of at most 32 that the footprint
    // reaches: bit ntx * row + column
    __device__ __forceinline__ unsigned tiles(int sh, int x0, int x1, int y0, int y1) const {
        const int tx0 = x0 >> sh, ty0 = y0 >> sh, ty1 = y1 >> sh, ntx = (x1 >> sh) - tx0 + 1;
        unsigned reached = 0u;
        int at = 0;
        for (int ty = ty0; ty <= ty1; ++ty, at += ntx) {
            int lo, hi;
            span(x0, x1, max(ty << sh, y0), min((ty << sh) + (1 << sh) - 1, y1), lo, hi);
            if (hi >= lo) reached |= ((2u << ((hi >> sh) - tx0)) - (1u << ((lo >> sh) - tx0))) << at;
        }
        return reached;
    }
    __device__ __forceinline__ TileRows from_lane(int src) const {
        TileRows q;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            q.s[k] = __shfl_sync(0xffffffffu, s[k], src);
            q.c[k] = __shfl_sync(0xffffffffu, c[k], src);
        }
        q.low = __shfl_sync(0xffffffffu, low, src);
        return q;
    }
};

// A warp visits the tiles of one box that a footprint reaches: a row per lane
// for the intervals, then the tiles of up to 32 rows dealt out evenly.  All
// lanes call it with the same box; visit(tx, ty) runs in the lanes that have one.
template <class Visit>
__device__ __forceinline__ void warp_tiles(const TileRows& rows, int sh, int x0, int x1, int y0, int y1, int lane,
                                           Visit visit) {
    const int ty0 = y0 >> sh, ty1 = y1 >> sh;
    for (int r = ty0; r <= ty1; r += 32) {
        const int ty = r + lane;
        int lo = 0, count = 0;
        if (ty <= ty1) {
            int hi;
            rows.span(x0, x1, max(ty << sh, y0), min((ty << sh) + (1 << sh) - 1, y1), lo, hi);
            count = hi >= lo ? (hi >> sh) - (lo >> sh) + 1 : 0;
            lo >>= sh;
        }
        int upto = count;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += v;
        }
        const int total = __shfl_sync(0xffffffffu, upto, 31), first = lo - (upto - count);
        for (int k0 = 0; k0 < total; k0 += 32) {
            const int k = k0 + lane;
            int row = 0;  // the first row whose tiles reach beyond k
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
                if (__shfl_sync(0xffffffffu, upto, row + o - 1) <= k) row += o;
            const int tx = __shfl_sync(0xffffffffu, first, row & 31) + k;
            if (k < total) visit(tx, r + row);
        }
    }
}

// bit n alone; 0 for n = 32 (the hardware shift saturates)
__device__ __forceinline__ unsigned bit_at(unsigned n) {
    unsigned r;
    asm("shl.b32 %0, 1, %1;" : "=r"(r) : "r"(n));
    return r;
}

// Rows of a 32 x 32 bit matrix (one per lane) to columns: lane i ends with
// bit j = lane j's bit i.  Five rounds of block swaps.
__device__ __forceinline__ unsigned transpose_bits(unsigned x, int lane) {
    unsigned m = 0x0000ffffu;
#pragma unroll
    for (int j = 16; j > 0; j >>= 1) {
        const unsigned y = __shfl_xor_sync(0xffffffffu, x, j);
        x = (lane & j) ? ((x & ~m) | ((y >> j) & m)) : ((x & m) | ((y << j) & ~m));
        m ^= m << (j >> 1);
    }
    return x;
}

// The pixels of a warp (RW rows of TS pixels; the first pixel is (X0, Y0))
// that a triangle can cover: its bounding box (x01, y01: first | last << 16)
// exactly, and its footprint edges (a, b, c) from the x interval that each
// leaves of a row, widened by kMaskSlack px in the edge's value (the float
// error of that value is below 0.03 px in the admitted coordinate range, and
// the reciprocal's far below that).  Bit r * TS + x is pixel (X0 + x, Y0 + r).
constexpr float kMaskSlack = 0.0625f;

template <int TS, int RW>
__device__ __forceinline__ unsigned pixel_mask(float a0, float b0, float c0, float a1, float b1, float c1, float a2,
                                               float b2, float c2, int x01, int y01, int X0, int Y0) {
    const int bx0 = max((x01 & 0xffff) - X0, 0), bx1 = min((x01 >> 16) - X0, TS - 1);
    const int by0 = (y01 & 0xffff) - Y0, by1 = (y01 >> 16) - Y0;
    if (bx1 < bx0 || by1 < 0 || by0 >= RW) return 0u;
    const float fx = X0 + 0.5f, fy = Y0 + 0.5f;
    const float ea[3] = {a0, a1, a2}, eb[3] = {b0, b1, b2}, ec[3] = {c0, c1, c2};
    // where edge k's value is -kMaskSlack in row r: x0 + r dx; the pixels right
    // of it (a > 0) or left of it remain, all of them where a is nearly 0
    float x0[3], dx[3];
    bool right[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float s = ea[k] * fx + eb[k] * fy + ec[k] + kMaskSlack, inv = __fdividef(-1.f, ea[k]);
        const bool bounds = fabsf(ea[k]) > 1e-6f;
        right[k] = !bounds || ea[k] > 0.f;
        x0[k] = bounds ? s * inv : -1.f;
        dx[k] = bounds ? eb[k] * inv : 0.f;
    }
    unsigned mask = 0u;
#pragma unroll
    for (int r = 0; r < RW; ++r) {
        float lo = (float)bx0, hi = (float)bx1;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float x = x0[k] + r * dx[k];
            if (right[k]) lo = fmaxf(lo, x);
            else hi = fminf(hi, x);
        }
        // ceil(lo) and floor(hi) + 1 by directed rounding at 2^23 (full-rate
        // additions; conversions run at a quarter of their rate)
        const unsigned l = __float_as_uint(__fadd_ru(fminf(lo, (float)TS), 8388608.f)) & 63u;
        const unsigned h = max(__float_as_uint(__fadd_rd(fmaxf(hi, -1.f), 8388609.f)) & 63u, l);
        if (r >= by0 && r <= by1) mask |= (bit_at(h) - bit_at(l)) << (r * TS);
    }
    return mask;
}

// Bilinear texture lookup at texel coordinates (x, y), texel centres at
// integer + 0.5, clamp-to-edge addressing: the four texels and weights.
struct BilinearTaps {
    long long i00, i10, i01, i11;
    float fx, fy;
};

__device__ __forceinline__ BilinearTaps bilinear_taps(float x, float y, int tw, int th) {
    const float sx = x - 0.5f, sy = y - 0.5f;
    const float x0f = floorf(sx), y0f = floorf(sy);
    BilinearTaps t;
    t.fx = sx - x0f;
    t.fy = sy - y0f;
    const int x0 = (int)x0f, y0 = (int)y0f;
    const int xa = min(max(x0, 0), tw - 1), xb = min(max(x0 + 1, 0), tw - 1);
    const int ya = min(max(y0, 0), th - 1), yb = min(max(y0 + 1, 0), th - 1);
    t.i00 = (long long)ya * tw + xa;
    t.i10 = (long long)ya * tw + xb;
    t.i01 = (long long)yb * tw + xa;
    t.i11 = (long long)yb * tw + xb;
    return t;
}

__device__ __forceinline__ float3 bilinear_sample(const float* T, const BilinearTaps& t) {
    const float3 c00 = ld3(T + 3 * t.i00), c10 = ld3(T + 3 * t.i10), c01 = ld3(T + 3 * t.i01), c11 = ld3(T + 3 * t.i11);
    const float w00 = (1.f - t.fx) * (1.f - t.fy), w10 = t.fx * (1.f - t.fy), w01 = (1.f - t.fx) * t.fy,
                w11 = t.fx * t.fy;
    return c00 * w00 + c10 * w10 + c01 * w01 + c11 * w11;
}

// One incident face of a vertex: the ids of its other two vertices in the
// face's order, and the vertex's own place in the face (0 to 2) in the top two
// bits of the second.  A fan walk reads one 8-byte entry and two vertices per
// face, where face ids would cost the id, three vertex ids and three vertices.
struct FanFace {
    int p, q, place;
    __device__ __forceinline__ explicit FanFace(int2 e) : p(e.x), q(e.y & 0x3fffffff), place((unsigned)e.y >> 30) {}
    // the face's three values in its order, from the own one and the others'
    template <class T>
    __device__ __forceinline__ void order(const T& own, const T& a, const T& b, T& v0, T& v1, T& v2) const {
        v0 = place == 0 ? own : a;
        v1 = place == 0 ? a : place == 1 ? own : b;
        v2 = place == 2 ? own : b;
    }
};

// the entry of vertex v for its face (a, b, c)
__host__ __device__ __forceinline__ int2 fan_entry(int v, int a, int b, int c) {
    const unsigned place = v == a ? 0u : v == b ? 1u : 2u;
    return make_int2(place == 0u ? b : a, (int)((unsigned)(place == 2u ? b : c) | place << 30));
}

// Sum of a vertex's incident face normals in increasing face order.
__device__ __forceinline__ float3 fan_normal(const float* __restrict__ P, const int2* __restrict__ fan, int2 range,
                                             int v) {
    const float3 own = ld3(P + 3 * v);
    float3 s = make_float3(0.f, 0.f, 0.f);
#pragma unroll 3
    for (int k = 0; k < range.y; ++k) {
        const FanFace f(fan[range.x + k]);
        const float3 a = ld3(P + 3 * f.p), b = ld3(P + 3 * f.q);
        float3 v0, v1, v2;
        f.order(own, a, b, v0, v1, v2);
        const float3 fn = cross(v1 - v0, v2 - v0);
        if (k == 0) {
            s = fn;
        } else {
            s.x = s.x + fn.x;
            s.y = s.y + fn.y;
            s.z = s.z + fn.z;
        }
    }
    return s;
}

// Second-order SH shading of an albedo (reference getShading,
// CudaRenderer/cpp/src/Utils/RendererUtil.h:135-173), one band set per channel.
__device__ __forceinline__ float sh_channel(const float* s, float3 d, float3 d2) {
    float r = s[0];
    r += s[1] * d.y;
    r += s[2] * d.z;
    r += s[3] * d.x;
    r += s[4] * (d.x * d.y);
    r += s[5] * (d.z * d.y);
    r += s[6] * (3.f * d2.z - 1.f);
    r += s[7] * (d.x * d.z);
    r += s[8] * (d2.x - d2.y);
    return r;
}

__device__ __forceinline__ float3 sh_illum(const float* sh, float3 n) {
    const float3 n2 = n * n;
    return make_float3(sh_channel(sh, n, n2), sh_channel(sh + 9, n, n2), sh_channel(sh + 18, n, n2));
}

struct Topology {
    int N = 0, F = 0;
    DevBuf mem[5];       // the arrays below, all in the first or each in its own
    DevPart faces;       // int3[F]
    DevPart fan;         // int2[3F]  vertex -> incident faces, increasing face id (FanFace)
    DevPart vf_id;       // int2[N]  (start, count)
    DevPart texcoords;   // float[6F]
    DevPart unit;        // float4[unit_frames * N]  normalised vertex normals of a UV map call
    int unit_frames = 0;
    bool has_texcoords = false;
};
// Frames whose normalised vertex normals have a place beside the topology: an
// allocation of their own makes an engine's first UV maps take 1.27 instead of
// 0.90 ms (40,962 vertices).
constexpr int kUnitFrames = 4;

// texel -> (face, barycentrics) table of the UV-space maps for one texture size
struct UvTable {
    int th = 0, tw = 0;
    bool valid = false;     // built by a call that ran (one recorded into a graph builds it at each replay)
    bool captured = false;  // a graph holds its address: it keeps its size and its texture size
    DevBuf buf;             // float4 per texel, then the int face per texel it is made from
};

struct UvTables {
    std::vector<UvTable> tables;  // one for each size that a graph holds, and at most one besides
    SpareBuf unit;  // normalised vertex normals of a call of more than Topology::unit_frames frames, 16 bytes each
    // the table of a texture size; the call has to build it unless it is valid
    hc_status get(int th, int tw, cudaStreamCaptureStatus capture, UvTable** out) {
        const bool recording = capture != cudaStreamCaptureStatusNone;
        const size_t need = (sizeof(float4) + sizeof(int)) * (size_t)th * tw;
        UvTable* t = nullptr;
        bool held = false;  // a table that a graph holds would have the room
        for (UvTable& k : tables) {
            if (k.th == th && k.tw == tw) {
                k.captured = k.captured || recording;
                *out = &k;
                return HC_OK;
            }
            if (!k.captured) t = &k;
            else held = held || k.buf.bytes >= need;
        }
        // under capture nothing is allocated, but for what another graph's table keeps from use
        const bool extra = recording && held && (!t || t->buf.bytes < need);
        if (!t || extra) {
            tables.emplace_back();
            t = &tables.back();
        }
        t->th = t->tw = 0;
        t->valid = false;
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        if (extra) HC_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
        const hc_status st = t->buf.ensure(need);
        if (extra) HC_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
        HC_TRY(st);
        t->th = th;
        t->tw = tw;
        t->captured = recording;
        *out = t;
        return HC_OK;
    }
};

// v / |v| (zero stays zero).  The contraction of |v|^2 is written out, so that
// every kernel gives the same values: a vertex normal's and a texel's differ in
// which of x^2 and y^2 is rounded first.
template <bool TEXEL>
__device__ __forceinline__ float3 unit_or_zero(float3 v) {
    const float l = sqrtf(TEXEL ? __fmaf_rn(v.z, v.z, __fmaf_rn(v.y, v.y, v.x * v.x))
                                : __fmaf_rn(v.z, v.z, __fmaf_rn(v.x, v.x, v.y * v.y)));
    return l != 0.f ? v / l : v;
}

// Work on a frame's mesh before any tile: vertex normals, triangle constants
// and projected vertices, one thread each.  They do not depend on one another,
// so one launch covers them, and ranges to fill, by its blocks in this order;
// a part without blocks is left out.
struct FrameSetup {
    int B, C, N, F;
    const int3* faces;
    const int2 *fan, *vf_id;
    const float* verts;
    float* vnormal;   // [B,C,N,3]
    float4* unit;     // with the normals: normalised, [B,N], or NULL
    TriFrame* tri;    // [B,F]
    const ViewCam* cams;
    float4* proj;     // [B*C,N]
    unsigned normal_blocks = 0, tri_blocks = 0, project_blocks = 0;
    FillRuns fills;
};
constexpr int kSetupThreads = 256, kViewThreads = 128;
__global__ void k_frame_setup(FrameSetup S);
// camera set-up, and ranges to fill by the blocks after the first view_blocks
__global__ void k_view_setup(int V, int C, const float* __restrict__ extr, const float* __restrict__ intr,
                             const CamLayout* __restrict__ layout, long long P_frame, long long T_frame,
                             long long Tb_frame, ViewCam* __restrict__ cams, int view_blocks, FillRuns fills);

// Optional per-kernel timing of the renderer (CUDA events around each
// launch on the launching stream), for benchmarks; off by default.
enum RendererKernel {
    kKViewSetup = 0, kKVertexNormals, kKTriFrame, kKBin, kKSpill, kKResolve, kKRenderGrad, kKNormalChain,
    kKCount
};

struct KernelClock {
    bool on = false, made = false;
    cudaEvent_t ev[2 * kKCount];
    unsigned recorded = 0;  // kernels with both events recorded since the last read
    void begin(int k, cudaStream_t s) {
        if (on) cudaEventRecord(ev[2 * k], s);
    }
    void end(int k, cudaStream_t s) {
        if (!on) return;
        cudaEventRecord(ev[2 * k + 1], s);
        recorded |= 1u << k;
    }
};

// The masked image L1 fused into the raster (hc_renderer_forward_l1 /
// hc_renderer_backward_l1): the forward's tile pass accumulates the loss of
// the pixels it shades, the adjoint forms the image gradient inline instead
// of reading it.
struct L1Fuse {
    const float* target = nullptr;        // [B, P_frame, 3]
    const unsigned char* mask = nullptr;  // [B, P_frame] foreground mask, or NULL
    L1State* state = nullptr;             // written by the forward, read by the adjoint
    float* loss = nullptr;                // forward: sum / count, or NULL
    const float* render = nullptr;        // adjoint: the forward's render buffer
};

struct RasterWorkspace {
    int cap_views = 0;   // views the buffers are sized for
    int tile = 16;
    int bin_cap = 512;
    // per-camera resolution and the device layout derived from it
    std::vector<int> cam_w, cam_h;
    int layout_tile = 0;                              // tile size the layout was built for
    long long P_frame = 0, T_frame = 0, Tb_frame = 0; // pixels / raster tiles / adjoint tiles per frame
    DevBuf layout, tile_cam, tile_cam_b;              // CamLayout[C]; camera of each tile of a frame
    long long spill_cap = 0;
    int spill_tile_cap = 0;
    DevBuf cams, tri_frame, tri_view, tile_state, bins, spill, spill_keys, stats;
    DevBuf proj;  // float4 [V,N]: projected vertices of the current call
    DevBuf claim;    // the tile resolve's tile counter
    DevBuf claim_b;  // the adjoint's tile counter
    // the adjoint's per-vertex gradient sums: once a call has needed them (floats
    // per frame, 0 before), sized with the cameras, so that they are replaced
    // only where those are
    DevBuf vacc;
    size_t vacc_floats = 0;
    hc_status size_vacc() {
        return vacc.ensure(sizeof(float) * vacc_floats * (cams.bytes / sizeof(ViewCam) / cam_w.size()));
    }
    int adjoint_dynamic = 1;  // the adjoint's tile schedule (hc_renderer_set_adjoint_schedule)
    KernelClock clock;
};

}  // namespace hc
