// Embedded-graph deformation (EmbeddedGraphGpu / EmbeddedGraphGpuGrad).
//
// Reference: CustomTensorFlowCPPOperators/src/CustomGPUOperators/EmbeddedGraphOperator/
// EmbeddedGraphGPUOp.cu:11-240 and EmbeddedGraphGPUOpGrad.cu:9-213, rotations from
// CustomTensorFlowCPPOperators/src/CudaUtils/EmbeddedGraphRotationHelper.h:53-210.
//
//   v_nr = sum_n w_n (R(delta_a_n) (v - g_n) + g_n + delta_t_n) + displacement
//   v'   = sum_s w_s (R(skinned_a_s) v_nr + skinned_t_s)
//
// with R(a) = Rz(a.z) Ry(a.y) Rx(a.x).  The reference re-evaluates both Euler
// rotations (6 sin/cos each) for every (vertex, node) pair; here a node pass
// evaluates them once per (frame, node) into a table the vertex pass gathers
// (1000 nodes x 96 B per frame stays in L1/L2).  The per-vertex arithmetic
// keeps the reference's operation order, so outputs match bit for bit.
//
// Adjoint: the displacement gradient u_v = (sum_s w_s R_s)^T g_v is computed
// once per vertex; node gradients gather u_v over the node -> vertex lists
// (no atomics):  dT_i = sum_v w_i u_v,  dA_i[k] = sum_v w_i (dR_i/da_k (v - g_i)) . u_v.
// In the reference mode the skinned gradients are zero (EmbeddedGraphGPUOpGrad.cu:
// 136-142); the full mode also returns them.
#include <algorithm>
#include <vector>

#include "eg_rot.cuh"
#include "hc_common.cuh"
#include "hc_math.cuh"
#include "renderer.cuh"  // FanFace

namespace hc {
namespace {

__device__ __forceinline__ float3 mtv(const float* M, float3 v) {  // M^T v, M row-major
    return make_float3(M[0] * v.x + M[3] * v.y + M[6] * v.z, M[1] * v.x + M[4] * v.y + M[7] * v.z,
                       M[2] * v.x + M[5] * v.y + M[8] * v.z);
}

// per (frame, node) table: R_delta (9), t_delta (3), R_skinned (9),
// t_skinned (3) and the node's base position g (3), 16-byte aligned so that a
// row of it is one vector load: rows 0-2 hold (R_delta, t_delta), rows 3-5
// (R_skinned, t_skinned), row 6 g
struct __align__(16) NodeRT {
    float rd[9];
    float td[3];
    float rs[9];
    float ts[3];
    float g[3];
    float pad;
};

__global__ void k_eg_nodes(int B, int M, const float* __restrict__ base, const int* __restrict__ node_vertex,
                           const float* __restrict__ dT, const float* __restrict__ dA, const float* __restrict__ sT,
                           const float* __restrict__ sA, NodeRT* __restrict__ tab, float* __restrict__ graph_out,
                           float* __restrict__ dA_copy, float* __restrict__ sA_copy) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= (long long)B * M) return;
    const int n = (int)(i % M);
    const float3 da = ld3(dA + 3 * i), sa = ld3(sA + 3 * i);
    const R33 Rd = euler_rot(da), Rs = euler_rot(sa);
    NodeRT t;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        t.rd[k] = Rd.m[k];
        t.rs[k] = Rs.m[k];
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        t.td[k] = dT[3 * i + k];
        t.ts[k] = sT[3 * i + k];
    }
    const float3 gb = ld3(base + 3LL * node_vertex[n]);
    t.g[0] = gb.x;
    t.g[1] = gb.y;
    t.g[2] = gb.z;
    t.pad = 0.f;
    tab[i] = t;
    if (dA_copy) st3(dA_copy + 3 * i, da);
    if (sA_copy) st3(sA_copy + 3 * i, sa);
    if (graph_out) {
        // deformed graph node (EmbeddedGraphGPUOp.cu:32-44)
        const float3 g = ld3(base + 3LL * node_vertex[n]);
        const float3 vnr = g + ld3(dT + 3 * i);
        const float3 d = mv(Rs, vnr) + ld3(sT + 3 * i);
        st3(graph_out + 3 * i, d);
    }
}

// The vertex pass, grid (vertex blocks, frames), a thread per vertex:
//   kEgForward      the deformed vertex (EmbeddedGraphGPUOp.cu:50-125)
//   kEgAdjoint      u_v = (sum_k w_k R_sk)^T g_v, the displacement gradient
//   kEgAdjointFull  u_v, and (u, g, v_nr, base vertex) packed in three 16-byte
//                   words per vertex for the node pass's gathers
// Sums in the reference's order: v_nr = sum_k w_k (R_dk (v - g_k) + g_k + t_dk)
// + disp, then sum_k w_k (R_sk v_nr + t_sk).
// Bound by the wavefronts of its gathers (28 16-byte loads per vertex at four
// nodes; copying a block's distinct nodes to shared memory first gained
// nothing: a block's vertices lie all over the mesh and share few nodes).  16
// frames x 40,962 vertices, 1000 nodes: 37 -> 33 us without the staging of the
// entries; the adjoint 60 -> 36 us, the outer sum it does not need left out and
// u_v formed in the same pass.
constexpr int kEgBlock = 128;
enum { kEgForward = 0, kEgAdjoint, kEgAdjointFull };
constexpr int kEgRows = sizeof(NodeRT) / sizeof(float4);

template <int MODE>
__global__ void __launch_bounds__(kEgBlock) k_eg_vertices(int N, int M, const float4* __restrict__ base4,
                                                          const int* __restrict__ poff, const int* __restrict__ pidx,
                                                          const float* __restrict__ pw,
                                                          const NodeRT* __restrict__ tab,
                                                          const float* __restrict__ disp,
                                                          const float* __restrict__ gv, float* __restrict__ out,
                                                          float4* __restrict__ packed) {
    const int b = blockIdx.y;
    const int v = blockIdx.x * kEgBlock + (int)threadIdx.x;
    if (v >= N) return;
    const float4* T = reinterpret_cast<const float4*>(tab + (long long)b * M);
    const long long i = (long long)b * N + v;
    const int off = poff[v], cnt = poff[v + 1] - off;
    auto weight = [&](int k) { return pw[off + k]; };
    auto row = [&](int k, int r) { return T[(long long)pidx[off + k] * kEgRows + r]; };
    auto rotation = [&](float4 a, float4 c, float4 d) {
        R33 R;
        R.m[0] = a.x;
        R.m[1] = a.y;
        R.m[2] = a.z;
        R.m[3] = a.w;
        R.m[4] = c.x;
        R.m[5] = c.y;
        R.m[6] = c.z;
        R.m[7] = c.w;
        R.m[8] = d.x;
        return R;
    };
    const float4 vb4 = base4[v];
    float3 vnr = make_float3(0.f, 0.f, 0.f);
    if constexpr (MODE != kEgAdjoint) {
        const float3 vb = make_float3(vb4.x, vb4.y, vb4.z);
        for (int k = 0; k < cnt; ++k) {
            const float w = weight(k);
            const float4 d = row(k, 2), gg = row(k, 6);
            const R33 R = rotation(row(k, 0), row(k, 1), d);
            const float3 g = make_float3(gg.x, gg.y, gg.z);
            vnr += w * (mv(R, vb - g) + g + make_float3(d.y, d.z, d.w));
        }
        vnr += ld3(disp + 3 * i);
    }
    if constexpr (MODE == kEgForward) {
        float3 dsum = make_float3(0.f, 0.f, 0.f);
        for (int k = 0; k < cnt; ++k) {
            const float w = weight(k);
            const float4 d = row(k, 5);
            const R33 R = rotation(row(k, 3), row(k, 4), d);
            dsum += w * (mv(R, vnr) + make_float3(d.y, d.z, d.w));
        }
        st3(out + 3 * i, dsum);
    } else {
        float S[9];
#pragma unroll
        for (int q = 0; q < 9; ++q) S[q] = 0.f;
        for (int k = 0; k < cnt; ++k) {
            const float w = weight(k);
            const R33 R = rotation(row(k, 3), row(k, 4), row(k, 5));
#pragma unroll
            for (int q = 0; q < 9; ++q) S[q] = S[q] + R.m[q] * w;
        }
        const float3 g = ld3(gv + 3 * i), u = mtv(S, g);
        st3(out + 3 * i, u);
        if constexpr (MODE == kEgAdjointFull) {
            packed[3 * i] = make_float4(u.x, u.y, u.z, vnr.x);
            packed[3 * i + 1] = make_float4(g.x, g.y, g.z, vnr.y);
            packed[3 * i + 2] = make_float4(vb4.x, vb4.y, vb4.z, vnr.z);
        }
    }
}

// normalised area-weighted normal of the deformed mesh (EmbeddedGraphGPUOp.cu:180-225)
__global__ void k_eg_normals(int B, int N, const int2* __restrict__ fan, const int2* __restrict__ vf_id,
                             const float* __restrict__ dv, float* __restrict__ out) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= (long long)B * N) return;
    const int b = (int)(i / N), v = (int)(i % N);
    st3(out + 3 * i, normalize3(fan_normal(dv + (long long)b * N * 3, fan, vf_id[v], v)));
}

// deformed markers (EmbeddedGraphGPUOp.cu:129-177)
__global__ void k_eg_markers(int B, int Mk, int M, const float* __restrict__ base, const int* __restrict__ node_vertex,
                             const float* __restrict__ markers, const int* __restrict__ m2n,
                             const NodeRT* __restrict__ tab, float* __restrict__ out) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= (long long)B * Mk) return;
    const int b = (int)(i / Mk), m = (int)(i % Mk);
    const int n = m2n[m];
    const NodeRT& T = tab[(long long)b * M + n];
    const float3 g = ld3(base + 3LL * node_vertex[n]);
    R33 Rd, Rs;
#pragma unroll
    for (int q = 0; q < 9; ++q) {
        Rd.m[q] = T.rd[q];
        Rs.m[q] = T.rs[q];
    }
    const float3 mnr = mv(Rd, ld3(markers + 3LL * m) - g) + g + make_float3(T.td[0], T.td[1], T.td[2]);
    st3(out + 3 * i, mv(Rs, mnr) + make_float3(T.ts[0], T.ts[1], T.ts[2]));
}

// ---------------------------------------------------------------------------
// adjoint
// ---------------------------------------------------------------------------

// Per (frame, node), a warp: gather over the node's vertices (and its marker).
// The gradient of an Euler angle is sum_v w (dR (v - g)) . u_v = dR : W with W =
// sum_v w u_v (v - g)^T, so the lanes sum the nine entries of W (12 operations
// per vertex instead of 45 for the three angles) and the angle derivatives
// enter once per node; FULL: the skinned gradients likewise from sum w g_v and
// sum w g_v v_nr^T, read from the vertices' packed values.  The 24 sums take
// one 31-shuffle reduction.  Bound by its gathers: 16 frames x 1000 nodes of
// 164 vertices 49 -> 34 us.
template <bool FULL>
__global__ void __launch_bounds__(256) k_eg_grad_node(
    int B, int N, int M, int Mk, const float4* __restrict__ base4, const int* __restrict__ node_vertex,
    const int* __restrict__ n2v_off, const int* __restrict__ n2v_size, const int* __restrict__ n2v_idx,
    const float* __restrict__ n2v_w, const int* __restrict__ n2m, const float* __restrict__ markers,
    const float* __restrict__ dA, const float* __restrict__ sA, const float* __restrict__ gm,
    const float* __restrict__ u, const float4* __restrict__ packed, const NodeRT* __restrict__ tab,
    float* __restrict__ gT, float* __restrict__ gA, float* __restrict__ gsT, float* __restrict__ gsA) {
    const long long i = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (i >= (long long)B * M) return;  // warp-uniform
    const int b = (int)(i / M), n = (int)(i % M);
    const float4 g4 = base4[node_vertex[n]];
    const float3 g = make_float3(g4.x, g4.y, g4.z);
    float a[32];  // t (3), W row-major (9); FULL: st (3), skinned W (9)
#pragma unroll
    for (int k = 0; k < 32; ++k) a[k] = 0.f;
    auto moment = [&](int at, float3 x, float3 y) {  // x, and x y^T
        a[at] += x.x;
        a[at + 1] += x.y;
        a[at + 2] += x.z;
        a[at + 3] += x.x * y.x;
        a[at + 4] += x.x * y.y;
        a[at + 5] += x.x * y.z;
        a[at + 6] += x.y * y.x;
        a[at + 7] += x.y * y.y;
        a[at + 8] += x.y * y.z;
        a[at + 9] += x.z * y.x;
        a[at + 10] += x.z * y.y;
        a[at + 11] += x.z * y.z;
    };
    const int off = n2v_off[n], cnt = n2v_size[n];
    for (int k = lane; k < cnt; k += 32) {
        const int v = n2v_idx[off + k];
        const float w = n2v_w[off + k];
        const long long vi = (long long)b * N + v;
        if constexpr (FULL) {
            const float4 q0 = packed[3 * vi], q1 = packed[3 * vi + 1], q2 = packed[3 * vi + 2];
            moment(0, w * make_float3(q0.x, q0.y, q0.z), make_float3(q2.x, q2.y, q2.z) - g);
            moment(12, w * make_float3(q1.x, q1.y, q1.z), make_float3(q0.w, q1.w, q2.w));
        } else {
            const float4 v4 = base4[v];
            moment(0, w * ld3(u + 3 * vi), make_float3(v4.x, v4.y, v4.z) - g);
        }
    }
    const int m = n2m ? n2m[n] : -1;
    if (lane == 0 && m >= 0 && gm) {
        // marker residual (EmbeddedGraphGPUOpGrad.cu:90-123): weight 1, its own node
        const NodeRT& T = tab[i];
        const float3 gmm = ld3(gm + 3 * ((long long)b * Mk + m));
        const float3 d = ld3(markers + 3LL * m) - g;
        moment(0, mtv(T.rs, gmm), d);
        if constexpr (FULL) {
            R33 Rd;
#pragma unroll
            for (int q = 0; q < 9; ++q) Rd.m[q] = T.rd[q];
            moment(12, gmm, mv(Rd, d) + g + make_float3(T.td[0], T.td[1], T.td[2]));
        }
    }
    const float sum = warp_sum32(a, lane);  // lane k: value k
    float r[24];
#pragma unroll
    for (int k = 0; k < (FULL ? 24 : 12); ++k) r[k] = __shfl_sync(0xffffffffu, sum, k);
    if (lane != 0) return;
    auto angle = [&](const R33& D, int at) {  // D : W
        float acc = 0.f;
#pragma unroll
        for (int q = 0; q < 9; ++q) acc += D.m[q] * r[at + q];
        return acc;
    };
    R33 d0, d1, d2;
    euler_rot_d(ld3(dA + 3 * i), d0, d1, d2);
    st3(gT + 3 * i, make_float3(r[0], r[1], r[2]));
    st3(gA + 3 * i, make_float3(angle(d0, 3), angle(d1, 3), angle(d2, 3)));
    float3 st = make_float3(0.f, 0.f, 0.f), sa = st;
    if constexpr (FULL) {
        euler_rot_d(ld3(sA + 3 * i), d0, d1, d2);
        st = make_float3(r[12], r[13], r[14]);
        sa = make_float3(angle(d0, 15), angle(d1, 15), angle(d2, 15));
    }
    st3(gsT + 3 * i, st);
    st3(gsA + 3 * i, sa);
}

}  // namespace
}  // namespace hc

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------
using namespace hc;

struct hc_eg_s {
    int N = 0, M = 0, Mk = 0, F = 0;
    int full_skinned_grad = 0;
    DevBuf base, node_vertex, n2v_off, n2v_size, n2v_idx, n2v_w;
    DevBuf base4, v2n_poff, v2n_pidx, v2n_pw;  // float4 base vertices; the vertex -> node CSR packed in vertex order
    DevBuf markers, m2n, n2m, fan, vf_id;
    DevBuf tab, packed;
    int reserved = 0;  // frames asked for with hc_eg_reserve
    // the packed vertices, which only the full skinned gradient reads
    hc_status reserve_packed(long long frames) {
        return full_skinned_grad ? packed.ensure(3 * sizeof(float4) * (size_t)frames * N) : HC_OK;
    }
};

static void release(hc_eg h) {
    DevBuf* bufs[] = {&h->base, &h->node_vertex, &h->n2v_off, &h->n2v_size, &h->n2v_idx, &h->n2v_w, &h->markers,
                      &h->m2n, &h->n2m, &h->fan, &h->vf_id, &h->tab, &h->packed, &h->base4, &h->v2n_poff,
                      &h->v2n_pidx, &h->v2n_pw};
    for (DevBuf* b : bufs) b->release();
    delete h;
}

namespace hc {
void build_vertex_faces(int N, const int32_t* faces, int F, std::vector<int>& vf, std::vector<int>& vf_id);
}

extern "C" hc_status hc_eg_create(hc_eg* out, int32_t n_vertices, const float* base_vertices, const int32_t* faces,
                                  int32_t n_faces, int32_t n_nodes, const int32_t* node_to_base_vertex,
                                  const int32_t* v2n_offsets, const int32_t* v2n_sizes, const int32_t* v2n_indices,
                                  const float* v2n_weights, const int32_t* n2v_offsets, const int32_t* n2v_sizes,
                                  const int32_t* n2v_indices, const float* n2v_weights, int32_t n_markers,
                                  const float* base_markers, const int32_t* marker_to_node) {
    clear_error();
    HC_REQUIRE(out, "out is NULL");
    *out = nullptr;
    HC_REQUIRE(n_vertices > 0 && n_nodes > 0 && n_faces > 0, "empty mesh or graph");
    HC_REQUIRE(base_vertices && faces && node_to_base_vertex && v2n_offsets && v2n_sizes && v2n_indices &&
                   v2n_weights && n2v_offsets && n2v_sizes && n2v_indices && n2v_weights,
               "NULL graph array");
    HC_REQUIRE(n_markers == 0 || (base_markers && marker_to_node), "markers need positions and node ids");
    HC_REQUIRE(n_vertices < (1 << 30), "too many vertices (%d)", n_vertices);
    long long nv2n = 0, nn2v = 0;
    for (int v = 0; v < n_vertices; ++v) {
        HC_REQUIRE(v2n_sizes[v] >= 0 && v2n_offsets[v] >= 0, "bad vertex->node range at %d", v);
        nv2n = std::max<long long>(nv2n, (long long)v2n_offsets[v] + v2n_sizes[v]);
    }
    for (int n = 0; n < n_nodes; ++n) {
        HC_REQUIRE(n2v_sizes[n] >= 0 && n2v_offsets[n] >= 0, "bad node->vertex range at %d", n);
        HC_REQUIRE(node_to_base_vertex[n] >= 0 && node_to_base_vertex[n] < n_vertices, "node %d vertex out of range",
                   n);
        nn2v = std::max<long long>(nn2v, (long long)n2v_offsets[n] + n2v_sizes[n]);
    }
    for (long long k = 0; k < nv2n; ++k)
        HC_REQUIRE(v2n_indices[k] >= 0 && v2n_indices[k] < n_nodes, "vertex->node index %d out of range",
                   v2n_indices[k]);
    for (long long k = 0; k < nn2v; ++k)
        HC_REQUIRE(n2v_indices[k] >= 0 && n2v_indices[k] < n_vertices, "node->vertex index %d out of range",
                   n2v_indices[k]);
    for (int i = 0; i < 3 * n_faces; ++i)
        HC_REQUIRE(faces[i] >= 0 && faces[i] < n_vertices, "face index out of range");
    std::vector<int> n2m(n_nodes, -1);
    for (int m = 0; m < n_markers; ++m) {
        HC_REQUIRE(marker_to_node[m] >= 0 && marker_to_node[m] < n_nodes, "marker %d node out of range", m);
        n2m[marker_to_node[m]] = m;
    }
    hc_eg_s* h = new hc_eg_s();
    h->N = n_vertices;
    h->M = n_nodes;
    h->Mk = n_markers;
    h->F = n_faces;
    std::vector<int> vf, vf_id;
    build_vertex_faces(n_vertices, faces, n_faces, vf, vf_id);
    std::vector<int2> fan(vf.size());
    for (int v = 0; v < n_vertices; ++v)
        for (int k = vf_id[2 * v]; k < vf_id[2 * v] + vf_id[2 * v + 1]; ++k)
            fan[k] = fan_entry(v, faces[3 * vf[k]], faces[3 * vf[k] + 1], faces[3 * vf[k] + 2]);
    hc_status st = HC_OK;
#define UP(buf, ptr, n)                                   \
    if (st == HC_OK) st = upload(h->buf, ptr, (size_t)(n));
    UP(base, base_vertices, 3LL * n_vertices);
    UP(node_vertex, node_to_base_vertex, n_nodes);
    UP(n2v_off, n2v_offsets, n_nodes);
    UP(n2v_size, n2v_sizes, n_nodes);
    UP(n2v_idx, n2v_indices, std::max<long long>(nn2v, 1));
    UP(n2v_w, n2v_weights, std::max<long long>(nn2v, 1));
    UP(n2m, n2m.data(), n_nodes);
    UP(fan, fan.data(), fan.size());
    UP(vf_id, vf_id.data(), vf_id.size());
    if (n_markers > 0) {
        UP(markers, base_markers, 3LL * n_markers);
        UP(m2n, marker_to_node, n_markers);
    }
    {
        // the vertex -> node lists packed contiguously in vertex order (a warp's
        // lists lie side by side), and the base vertices padded to float4
        std::vector<int> poff((size_t)n_vertices + 1, 0), pidx;
        std::vector<float> pw;
        std::vector<float4> b4((size_t)n_vertices);
        for (int v = 0; v < n_vertices; ++v) {
            for (int k = 0; k < v2n_sizes[v]; ++k) {
                pidx.push_back(v2n_indices[v2n_offsets[v] + k]);
                pw.push_back(v2n_weights[v2n_offsets[v] + k]);
            }
            poff[v + 1] = (int)pidx.size();
            b4[v] = make_float4(base_vertices[3 * v], base_vertices[3 * v + 1], base_vertices[3 * v + 2], 0.f);
        }
        if (pidx.empty()) {
            pidx.push_back(0);
            pw.push_back(0.f);
        }
        UP(v2n_poff, poff.data(), poff.size());
        UP(v2n_pidx, pidx.data(), pidx.size());
        UP(v2n_pw, pw.data(), pw.size());
        UP(base4, b4.data(), b4.size());
    }
#undef UP
    if (st != HC_OK) {
        release(h);
        return st;
    }
    *out = h;
    return HC_OK;
}

extern "C" hc_status hc_eg_destroy(hc_eg h) {
    clear_error();
    if (h) release(h);
    return HC_OK;
}

extern "C" hc_status hc_eg_set_full_skinned_gradient(hc_eg h, int32_t enable) {
    clear_error();
    HC_REQUIRE(h, "invalid handle");
    h->full_skinned_grad = enable ? 1 : 0;
    return h->reserve_packed(h->reserved);
}

extern "C" hc_status hc_eg_reserve(hc_eg h, int32_t batch) {
    clear_error();
    HC_REQUIRE(h && batch > 0, "invalid handle or batch");
    HC_TRY(h->tab.ensure(sizeof(NodeRT) * (size_t)batch * h->M));
    h->reserved = std::max(h->reserved, batch);
    return h->reserve_packed(h->reserved);
}

// the vertex pass over B frames, at most 65535 (the grid's limit) at a time
template <int MODE>
static hc_status launch_vertices(hc_eg h, cudaStream_t s, int B, const float* disp, const float* gv, float* out) {
    for (int b = 0; b < B; b += 65535) {
        const size_t at = 3 * (size_t)b * h->N;
        k_eg_vertices<MODE><<<dim3(div_up(h->N, kEgBlock), std::min(B - b, 65535)), kEgBlock, 0, s>>>(
            h->N, h->M, h->base4.as<float4>(), h->v2n_poff.as<int>(), h->v2n_pidx.as<int>(), h->v2n_pw.as<float>(),
            h->tab.as<NodeRT>() + (size_t)b * h->M, disp ? disp + at : nullptr, gv ? gv + at : nullptr, out + at,
            h->packed.as<float4>() + at);
        HC_CHECK_LAUNCH();
    }
    return HC_OK;
}

extern "C" hc_status hc_eg_forward(hc_eg h, void* stream, int32_t batch, const float* nodes_delta_translation,
                                   const float* nodes_delta_rotation, const float* nodes_skinned_translation,
                                   const float* nodes_skinned_rotation, const float* vertex_displacements,
                                   float* deformed_vertices, float* deformed_normals, float* deformed_markers,
                                   float* deformed_graph, float* d_delta_rotation, float* d_skinned_rotation) {
    clear_error();
    HC_REQUIRE(h, "invalid handle");
    HC_REQUIRE(batch > 0, "batch must be positive");
    HC_REQUIRE(nodes_delta_translation && nodes_delta_rotation && nodes_skinned_translation &&
                   nodes_skinned_rotation && vertex_displacements && deformed_vertices,
               "NULL input/output pointer");
    HC_REQUIRE(h->Mk == 0 || deformed_markers, "deformed_markers output missing");
    cudaStream_t s = (cudaStream_t)stream;
    HC_TRY(h->tab.ensure(sizeof(NodeRT) * (size_t)batch * h->M));
    NodeRT* tab = h->tab.as<NodeRT>();
    const long long BM = (long long)batch * h->M, BN = (long long)batch * h->N;
    k_eg_nodes<<<div_up(BM, 128), 128, 0, s>>>(batch, h->M, h->base.as<float>(), h->node_vertex.as<int>(),
                                               nodes_delta_translation, nodes_delta_rotation,
                                               nodes_skinned_translation, nodes_skinned_rotation, tab, deformed_graph,
                                               d_delta_rotation, d_skinned_rotation);
    HC_CHECK_LAUNCH();
    HC_REQUIRE(batch <= 65535, "too many frames in one call (%d)", batch);
    HC_TRY(launch_vertices<kEgForward>(h, s, batch, vertex_displacements, nullptr, deformed_vertices));
    if (deformed_normals) {
        k_eg_normals<<<div_up(BN, 128), 128, 0, s>>>(batch, h->N, h->fan.as<int2>(), h->vf_id.as<int2>(),
                                                     deformed_vertices, deformed_normals);
        HC_CHECK_LAUNCH();
    }
    if (h->Mk > 0) {
        k_eg_markers<<<div_up((long long)batch * h->Mk, 128), 128, 0, s>>>(
            batch, h->Mk, h->M, h->base.as<float>(), h->node_vertex.as<int>(), h->markers.as<float>(),
            h->m2n.as<int>(), tab, deformed_markers);
        HC_CHECK_LAUNCH();
    }
    return HC_OK;
}

extern "C" hc_status hc_eg_backward(hc_eg h, void* stream, int32_t batch, const float* deformed_vertices_grad,
                                    const float* deformed_markers_grad, const float* d_delta_a,
                                    const float* d_skinned_a, float* nodes_t_grad, float* nodes_r_grad,
                                    float* nodes_skinned_t_grad, float* nodes_skinned_r_grad,
                                    float* vertex_displacements_grad, const float* nodes_delta_translation,
                                    const float* vertex_displacements) {
    clear_error();
    HC_REQUIRE(h, "invalid handle");
    HC_REQUIRE(batch > 0, "batch must be positive");
    HC_REQUIRE(deformed_vertices_grad && d_delta_a && d_skinned_a && nodes_t_grad && nodes_r_grad &&
                   nodes_skinned_t_grad && nodes_skinned_r_grad && vertex_displacements_grad,
               "NULL input/output pointer");
    const bool full = h->full_skinned_grad != 0;
    HC_REQUIRE(!full || (nodes_delta_translation && vertex_displacements),
               "the full skinned gradient needs nodes_delta_translation and vertex_displacements");
    cudaStream_t s = (cudaStream_t)stream;
    HC_TRY(h->tab.ensure(sizeof(NodeRT) * (size_t)batch * h->M));
    const long long BM = (long long)batch * h->M;
    NodeRT* tab = h->tab.as<NodeRT>();
    // node table from the saved angles; the backward reads the rotations, and
    // (full mode) the delta translations -- the skinned-translation slot of
    // the table is unused here, so it is filled from the same array
    k_eg_nodes<<<div_up(BM, 128), 128, 0, s>>>(batch, h->M, h->base.as<float>(), h->node_vertex.as<int>(),
                                               full ? nodes_delta_translation : d_delta_a, d_delta_a,
                                               full ? nodes_delta_translation : d_delta_a, d_skinned_a, tab, nullptr,
                                               nullptr, nullptr);
    HC_CHECK_LAUNCH();
    if (full) {
        HC_REQUIRE(batch <= 65535, "too many frames in one call (%d)", batch);
        HC_TRY(h->reserve_packed(batch));
        HC_TRY(launch_vertices<kEgAdjointFull>(h, s, batch, vertex_displacements, deformed_vertices_grad,
                                               vertex_displacements_grad));
    } else {
        HC_TRY(launch_vertices<kEgAdjoint>(h, s, batch, nullptr, deformed_vertices_grad, vertex_displacements_grad));
    }
    auto kernel = full ? k_eg_grad_node<true> : k_eg_grad_node<false>;
    kernel<<<div_up(BM * 32, 256), 256, 0, s>>>(
        batch, h->N, h->M, h->Mk, h->base4.as<float4>(), h->node_vertex.as<int>(), h->n2v_off.as<int>(),
        h->n2v_size.as<int>(), h->n2v_idx.as<int>(), h->n2v_w.as<float>(), h->n2m.as<int>(), h->markers.as<float>(),
        d_delta_a, d_skinned_a, deformed_markers_grad, vertex_displacements_grad, h->packed.as<float4>(), tab,
        nodes_t_grad, nodes_r_grad, nodes_skinned_t_grad, nodes_skinned_r_grad);
    HC_CHECK_LAUNCH();
    return HC_OK;
}
