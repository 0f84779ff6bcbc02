// UV-space maps of the renderer (compute_normal_map = normal / position / face).
//
// Reference: CudaRenderer/cpp/src/Renderer/CUDABasedRasterization.cpp:187-330
// (texel table, built on the host with OpenMP on the first forward call) and
// CUDABasedRasterization.cu:458-549 (renderNormalMapDevice).  In these modes
// the reference op does not rasterise the views at all: the face, barycentric
// and render buffers keep their initial values (-1, 0, 0) and only the vertex
// normals and the UV map are written (CUDABasedRasterization.cu:562-575).
//
// The texel table maps every texel centre to the triangle whose UV triangle
// contains it and the barycentrics of the texel in that triangle.  Here it is
// built on the device, once per texture size: one thread per triangle visits
// the texels of its UV bounding box (widened by 2 texels, as in the
// reference) with the reference's host ray test, keeping the largest face id
// per texel (the last writer of the reference's loop in serial order; its
// OpenMP loop leaves texels on shared UV edges to whichever thread writes
// last), then one thread per texel recomputes the barycentrics of the winner.
// The host ray test runs without fused multiply-adds (x86-64 SSE code), so
// its arithmetic is written here with explicitly rounded single operations.
#include <algorithm>

#include "renderer.cuh"

namespace hc {
namespace {

// host float arithmetic: every product and sum rounded on its own
struct HF3 {
    float x, y, z;
};
__device__ __forceinline__ HF3 hf3(float x, float y, float z) { return HF3{x, y, z}; }
__device__ __forceinline__ HF3 hsub(HF3 a, HF3 b) { return hf3(__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z)); }
__device__ __forceinline__ HF3 hadd(HF3 a, HF3 b) { return hf3(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y), __fadd_rn(a.z, b.z)); }
__device__ __forceinline__ HF3 hscale(float s, HF3 a) { return hf3(__fmul_rn(s, a.x), __fmul_rn(s, a.y), __fmul_rn(s, a.z)); }
__device__ __forceinline__ HF3 hdiv(HF3 a, float s) { return hf3(__fdiv_rn(a.x, s), __fdiv_rn(a.y, s), __fdiv_rn(a.z, s)); }
__device__ __forceinline__ float hdot(HF3 a, HF3 b) {
    return __fadd_rn(__fadd_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)), __fmul_rn(a.z, b.z));
}
__device__ __forceinline__ HF3 hcross(HF3 a, HF3 b) {
    return hf3(__fsub_rn(__fmul_rn(a.y, b.z), __fmul_rn(a.z, b.y)), __fsub_rn(__fmul_rn(a.z, b.x), __fmul_rn(a.x, b.z)),
               __fsub_rn(__fmul_rn(a.x, b.y), __fmul_rn(a.y, b.x)));
}

// rayTriangleIntersectHost (CUDABasedRasterization.cpp:187-262) for the
// texel ray: origin (x + 0.5, y + 0.5, 1), direction (0, 0, -1), triangle in
// texel units with z = 0.
__device__ bool texel_hit(HF3 o, HF3 v0, HF3 v1, HF3 v2, float& a, float& b) {
    v0 = hdiv(v0, 1000.f);
    v1 = hdiv(v1, 1000.f);
    v2 = hdiv(v2, 1000.f);
    o = hdiv(o, 1000.f);
    const HF3 dir = hf3(0.f, 0.f, -1.f);
    const HF3 N = hcross(hsub(v1, v0), hsub(v2, v0));
    const float ndr = hdot(dir, N);
    if (fabsf(ndr) < 0.0000001f) return false;
    const float t = __fdiv_rn(__fsub_rn(hdot(v0, N), hdot(o, N)), ndr);
    if (t < 0.f) return false;
    const HF3 P = hadd(o, hscale(t, dir));
    if (hdot(N, hcross(hsub(v1, v0), hsub(P, v0))) < 0.f) return false;
    if ((a = hdot(N, hcross(hsub(v2, v1), hsub(P, v1)))) < 0.f) return false;
    if ((b = hdot(N, hcross(hsub(v0, v2), hsub(P, v2)))) < 0.f) return false;
    const float denom = hdot(N, N);
    a = __fdiv_rn(a, denom);
    b = __fdiv_rn(b, denom);
    return true;
}

__device__ __forceinline__ void uv_corners(const float* tc, int f, int tw, int th, HF3& t0, HF3& t1, HF3& t2) {
    const float* c = tc + 6LL * f;
    t0 = hf3(__fmul_rn((float)tw, c[0]), __fmul_rn((float)th, __fsub_rn(1.f, c[1])), 0.f);
    t1 = hf3(__fmul_rn((float)tw, c[2]), __fmul_rn((float)th, __fsub_rn(1.f, c[3])), 0.f);
    t2 = hf3(__fmul_rn((float)tw, c[4]), __fmul_rn((float)th, __fsub_rn(1.f, c[5])), 0.f);
}

__global__ void k_texel_faces(int F, int tw, int th, const float* __restrict__ tc, int* __restrict__ texel_face) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= F) return;
    HF3 t0, t1, t2;
    uv_corners(tc, f, tw, th, t0, t1, t2);
    const int x0 = (int)fmaxf(fminf(t0.x, fminf(t1.x, t2.x)) - 2.f, 0.f);
    const int x1 = (int)fminf(fmaxf(t0.x, fmaxf(t1.x, t2.x)) + 2.f, (float)tw);
    const int y0 = (int)fmaxf(fminf(t0.y, fminf(t1.y, t2.y)) - 2.f, 0.f);
    const int y1 = (int)fminf(fmaxf(t0.y, fmaxf(t1.y, t2.y)) + 2.f, (float)th);
    for (int x = x0; x < x1; ++x)
        for (int y = y0; y < y1; ++y) {
            float a, b;
            if (texel_hit(hf3(x + 0.5f, y + 0.5f, 1.f), t0, t1, t2, a, b)) atomicMax(texel_face + y * tw + x, f);
        }
}

// (face, a, b, c) per texel; (0, 0, 0, 0) where no triangle covers it
__global__ void k_texel_table(int tw, int th, const float* __restrict__ tc, const int* __restrict__ texel_face,
                              float4* __restrict__ table) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= tw * th) return;
    const int f = texel_face[i];
    float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
    if (f >= 0) {
        HF3 t0, t1, t2;
        uv_corners(tc, f, tw, th, t0, t1, t2);
        float a = 0.f, b = 0.f;
        texel_hit(hf3(i % tw + 0.5f, i / tw + 0.5f, 1.f), t0, t1, t2, a, b);
        r = make_float4((float)f, a, b, __fsub_rn(__fsub_rn(1.f, a), b));
    }
    table[i] = r;
}

// v0 a + v1 b + v2 c, its contraction written out: the same values in every kernel
__device__ __forceinline__ float blend1(float a, float b, float c, float4 t) {
    return __fmaf_rn(c, t.w, __fmaf_rn(a, t.y, b * t.z));
}
__device__ __forceinline__ float3 blend(float3 a, float3 b, float3 c, float4 t) {
    return make_float3(blend1(a.x, b.x, c.x, t), blend1(a.y, b.y, c.y, t), blend1(a.z, b.z, c.z, t));
}

// renderNormalMapDevice (CUDABasedRasterization.cu:458-549) per (frame, texel):
// normal = barycentric blend of the normalised vertex normals of camera 0,
// normalised; position = blend of the vertex positions; face = the face id.
// A thread takes one texel of kUvFrames frames: the table entry and the face's
// ids are read once for them.  unit: the vertex normals already normalised, one
// 16-byte load each (k_frame_setup; 40,962 normalisations instead of three per
// texel); NULL: from vnormal.  512^2 texels, 81,920 triangles, 4 frames: 17.0 us
// without either, 13.5 with the unit normals, 9.8 with four frames per thread
// too (1, 2, 3 and 16 frames: 4.9, 7.8, 10.7 and 46.6 us -> 5.0, 6.6, 8.2 and 28.3).
constexpr int kUvFrames = 4;
__global__ void k_uv_map(int B, int C, int N, int n_texels, int mode, const int3* __restrict__ faces,
                         const float4* __restrict__ table, const float* __restrict__ verts,
                         const float* __restrict__ vnormal, const float4* __restrict__ unit,
                         float* __restrict__ out) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n_texels) return;
    const float4 info = table[p];
    const int3 id = mode == kNmFace ? make_int3(0, 0, 0) : faces[(int)info.x];
    for (int b0 = blockIdx.y * kUvFrames; b0 < B; b0 += gridDim.y * kUvFrames) {
#pragma unroll
        for (int k = 0; k < kUvFrames; ++k) {
            const int b = b0 + k;
            if (b >= B) break;
            float3 r;
            if (mode == kNmFace) {
                r = make_float3(info.x, info.x, info.x);
            } else {
                float3 v0, v1, v2;
                if (mode == kNmOriginal && unit) {
                    const float4* u = unit + (long long)b * N;
                    const float4 u0 = u[id.x], u1 = u[id.y], u2 = u[id.z];
                    v0 = make_float3(u0.x, u0.y, u0.z);
                    v1 = make_float3(u1.x, u1.y, u1.z);
                    v2 = make_float3(u2.x, u2.y, u2.z);
                } else {
                    const float* src =
                        mode == kNmOriginal ? vnormal + (long long)b * C * N * 3 : verts + (long long)b * N * 3;
                    v0 = ld3(src + 3 * id.x), v1 = ld3(src + 3 * id.y), v2 = ld3(src + 3 * id.z);
                    if (mode == kNmOriginal) {
                        v0 = unit_or_zero<false>(v0);
                        v1 = unit_or_zero<false>(v1);
                        v2 = unit_or_zero<false>(v2);
                    }
                }
                r = blend(v0, v1, v2, info);
                if (mode == kNmOriginal) r = unit_or_zero<true>(r);
            }
            st3(out + 3 * ((long long)b * n_texels + p), r);
        }
    }
}

}  // namespace

hc_status raster_uv_maps(const Topology& topo, UvTables& tab, cudaStream_t s, int B, int C, long long P_frame, int mode,
                         const float* verts, int tex_h, int tex_w, float* bary, int* face, float* render,
                         float* vnormal, float* uv_map) {
    HC_REQUIRE(topo.has_texcoords, "compute_normal_map needs texture_coordinates");
    HC_REQUIRE(tex_h > 0 && tex_w > 0, "compute_normal_map needs the texture size");
    HC_REQUIRE(uv_map, "compute_normal_map needs the normal_map output");
    const long long px = (long long)B * P_frame;
    const int N = topo.N, F = topo.F;
    FrameSetup S{};
    S.B = B;
    S.C = C;
    S.N = N;
    S.F = F;
    S.fan = topo.fan.as<int2>();
    S.vf_id = topo.vf_id.as<int2>();
    S.verts = verts;
    S.vnormal = vnormal;
    // without room for them the normals are normalised where they are used
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    HC_CUDA(cudaStreamIsCapturing(s, &capture));
    if (mode == kNmOriginal) {
        if (B <= topo.unit_frames) S.unit = topo.unit.as<float4>();
        else if (tab.unit.room(sizeof(float4) * (size_t)B * N, capture)) S.unit = tab.unit.as<float4>();
    }
    S.fills.add(face, sizeof(int) * (size_t)px, 0xff);
    S.fills.add(bary, sizeof(float) * 2 * (size_t)px);
    S.fills.add(render, sizeof(float) * 3 * (size_t)px);
    S.normal_blocks = div_up((long long)B * N, kSetupThreads);
    k_frame_setup<<<S.normal_blocks + S.fills.blocks(kSetupThreads), kSetupThreads, 0, s>>>(S);
    HC_CHECK_LAUNCH();
    const int nt = tex_h * tex_w;
    UvTable* table = nullptr;
    HC_TRY(tab.get(tex_h, tex_w, capture, &table));
    float4* texels = table->buf.as<float4>();
    if (!table->valid) {
        int* texel_face = reinterpret_cast<int*>(texels + nt);  // one allocation for both
        HC_CUDA(cudaMemsetAsync(texel_face, 0xff, sizeof(int) * (size_t)nt, s));
        k_texel_faces<<<div_up(F, 128), 128, 0, s>>>(F, tex_w, tex_h, topo.texcoords.as<float>(), texel_face);
        HC_CHECK_LAUNCH();
        k_texel_table<<<div_up(nt, 256), 256, 0, s>>>(tex_w, tex_h, topo.texcoords.as<float>(), texel_face, texels);
        HC_CHECK_LAUNCH();
        table->valid = capture == cudaStreamCaptureStatusNone;
    }
    k_uv_map<<<dim3(div_up(nt, 256), std::min(div_up(B, kUvFrames), 65535)), 256, 0, s>>>(
        B, C, N, nt, mode, topo.faces.as<int3>(), texels, verts, vnormal, S.unit, uv_map);
    HC_CHECK_LAUNCH();
    return HC_OK;
}

}  // namespace hc
