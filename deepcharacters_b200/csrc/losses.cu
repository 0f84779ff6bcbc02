// Image loss of the training step: masked L1 on 255-scaled colours, divided
// by the number of non-zero residual entries (Projects/HoloportedCharacters/
// HPCMeshDL.py:669-688: difference = 255 (R - T) * mask * model_mask,
// loss = sum |difference| / count_nonzero(difference)), and its gradient
// d loss / d R = 255 sign(difference) * mask * model_mask / count
// (the count is a constant for the gradient, as in TF).
#include <algorithm>
#include <math.h>

#include "hc_common.cuh"
#include "hc_math.cuh"

namespace hc {
namespace {

using L1Acc = L1State;

__global__ void k_l1_reduce(long long n_px, const float* __restrict__ render, const float* __restrict__ target,
                            const int* __restrict__ face, const unsigned char* __restrict__ mask,
                            L1Acc* __restrict__ acc) {
    float s = 0.f;
    unsigned cnt = 0;
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n_px;
         p += (long long)gridDim.x * blockDim.x) {
        const bool m = face[p] >= 0 && (!mask || mask[p]);
        if (!m) continue;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float d = l1_diff(render[3 * p + c], target[3 * p + c]);
            s += fabsf(d);
            cnt += d != 0.f;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, o);
        cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    }
    __shared__ float ss[32];
    __shared__ unsigned sc[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) {
        ss[w] = s;
        sc[w] = cnt;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0;
        unsigned long long c = 0;
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) {
            t += ss[i];
            c += sc[i];
        }
        atomicAdd(&acc->sum, t);
        atomicAdd(&acc->count, c);
    }
}

__global__ void k_l1_grad(long long n_px, const float* __restrict__ render, const float* __restrict__ target,
                          const int* __restrict__ face, const unsigned char* __restrict__ mask,
                          const L1Acc* __restrict__ acc, float* __restrict__ grad, float* __restrict__ loss) {
    const unsigned long long cnt = acc->count;
    const float scale = cnt ? 255.f / (float)cnt : 0.f;
    if (blockIdx.x == 0 && threadIdx.x == 0 && loss) *loss = cnt ? (float)(acc->sum / (double)cnt) : 0.f;
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n_px;
         p += (long long)gridDim.x * blockDim.x) {
        const bool m = face[p] >= 0 && (!mask || mask[p]);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            float g = 0.f;
            if (m) {
                g = l1_grad(l1_diff(render[3 * p + c], target[3 * p + c]), scale);
            }
            grad[3 * p + c] = g;
        }
    }
}

// The loss and its gradient with a byte of scratch per pixel: the first pass
// reads the images once, four pixels per thread in 16-byte loads, and leaves
// the signs of a pixel's differences (bits 2c, 2c+1: channel c positive,
// negative) beside the sums; the second forms the gradient from the signs and
// the count.  Reading the images again instead costs 28 bytes per pixel.
// Bound by HBM: 28 bytes read and 12 written per pixel (and one byte each way,
// mostly in L2).  8 x 1024^2: 65 us for both, the pair above 115 us.
__global__ void __launch_bounds__(256) k_l1_signs(long long n_px, const float4* __restrict__ render,
                                                  const float4* __restrict__ target, const int4* __restrict__ face,
                                                  const unsigned char* __restrict__ mask, L1Acc* __restrict__ acc,
                                                  unsigned char* __restrict__ signs) {
    float s = 0.f;
    unsigned cnt = 0;
    const float* rf = reinterpret_cast<const float*>(render);
    const float* tf = reinterpret_cast<const float*>(target);
    const int* ff = reinterpret_cast<const int*>(face);
    auto term = [&](float r, float t, int c) -> unsigned {
        const float d = l1_diff(r, t);
        s += fabsf(d);
        cnt += d != 0.f;
        return (d > 0.f ? 1u : d < 0.f ? 2u : 0u) << (2 * c);
    };
    const long long n4 = n_px / 4, stride = (long long)gridDim.x * blockDim.x;
    const long long first = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    for (long long i = first; i < n4; i += stride) {
        const int4 f = face[i];
        const uchar4 m = mask ? make_uchar4(mask[4 * i], mask[4 * i + 1], mask[4 * i + 2], mask[4 * i + 3])
                              : make_uchar4(1, 1, 1, 1);
        const bool on[4] = {f.x >= 0 && m.x, f.y >= 0 && m.y, f.z >= 0 && m.z, f.w >= 0 && m.w};
        unsigned code[4] = {0u, 0u, 0u, 0u};
        if (on[0] || on[1] || on[2] || on[3]) {
            float r[12], t[12];
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const float4 a = render[3 * i + q], b = target[3 * i + q];
                r[4 * q] = a.x, r[4 * q + 1] = a.y, r[4 * q + 2] = a.z, r[4 * q + 3] = a.w;
                t[4 * q] = b.x, t[4 * q + 1] = b.y, t[4 * q + 2] = b.z, t[4 * q + 3] = b.w;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (on[k])
#pragma unroll
                    for (int c = 0; c < 3; ++c) code[k] |= term(r[3 * k + c], t[3 * k + c], c);
        }
        reinterpret_cast<uchar4*>(signs)[i] = make_uchar4(code[0], code[1], code[2], code[3]);
    }
    for (long long p = 4 * n4 + first; p < n_px; p += stride) {
        unsigned code = 0;
        if (ff[p] >= 0 && (!mask || mask[p]))
            for (int c = 0; c < 3; ++c) code |= term(rf[3 * p + c], tf[3 * p + c], c);
        signs[p] = (unsigned char)code;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, o);
        cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    }
    __shared__ float ss[8];
    __shared__ unsigned sc[8];
    if ((threadIdx.x & 31) == 0) {
        ss[threadIdx.x >> 5] = s;
        sc[threadIdx.x >> 5] = cnt;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0;
        unsigned long long c = 0;
        for (int i = 0; i < 8; ++i) {
            t += ss[i];
            c += sc[i];
        }
        atomicAdd(&acc->sum, t);
        atomicAdd(&acc->count, c);
    }
}

// four channels' gradients from their signs (2 bits each)
__device__ __forceinline__ float4 signed_scale(unsigned bits, float scale) {
    float g[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const unsigned c = (bits >> (2 * k)) & 3u;
        g[k] = c == 1u ? scale : c == 2u ? -scale : 0.f;
    }
    return make_float4(g[0], g[1], g[2], g[3]);
}

// A warp takes 128 pixels: a lane loads the signs of four (24 bits), and each 16
// bytes of the gradient are one byte of those, handed over by a shuffle, so that
// the loads and the stores are both consecutive; the signs of the warp's next
// pixels are loaded before this one's stores.  Bound by HBM (12 bytes per pixel
// written).  A thread per 16 bytes loading its own two signs -> this: 8 x 1024^2
// 26.6 -> 19.7 us.
__global__ void __launch_bounds__(256) k_l1_from_signs(long long n, const unsigned char* __restrict__ signs,
                                                       const L1Acc* __restrict__ acc, float4* __restrict__ grad,
                                                       float* __restrict__ loss) {
    const unsigned long long cnt = acc->count;
    const float scale = cnt ? 255.f / (float)cnt : 0.f;
    if (blockIdx.x == 0 && threadIdx.x == 0 && loss) *loss = cnt ? (float)(acc->sum / (double)cnt) : 0.f;
    const int lane = threadIdx.x & 31;
    const long long n_px = n / 3, groups = n_px >> 7, warps = (long long)gridDim.x * (blockDim.x >> 5);
    const uchar4* s4 = reinterpret_cast<const uchar4*>(signs);
    long long g = blockIdx.x * (long long)(blockDim.x >> 5) + (threadIdx.x >> 5);
    uchar4 next = g < groups ? s4[32 * g + lane] : make_uchar4(0, 0, 0, 0);
    for (; g < groups; g += warps) {
        const unsigned mine = next.x | next.y << 6 | next.z << 12 | next.w << 18;
        if (g + warps < groups) next = s4[32 * (g + warps) + lane];
#pragma unroll
        for (int t = 0; t < 3; ++t) {
            const unsigned j = lane + 32 * t;  // the 16 bytes j of the group
            grad[96 * g + j] = signed_scale(__shfl_sync(0xffffffffu, mine, j / 3) >> (8 * (j % 3)), scale);
        }
    }
    // the pixels beyond the last full group
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long p = 128 * groups + i;
    if (i < 128 && p < n_px) {
        const float4 v = signed_scale(signs[p], scale);
        float* out = reinterpret_cast<float*>(grad) + 3 * p;
        out[0] = v.x, out[1] = v.y, out[2] = v.z;
    }
}

// one pass: grad = 2 w x and the block partials of sum x^2 (vec: 16-byte
// loads and stores, n a multiple of 4 and both pointers 16-byte aligned)
__global__ void k_sumsq_fused(long long n, const float* __restrict__ x, float weight, double* __restrict__ acc,
                              float* __restrict__ grad, int vec) {
    const float k = 2.f * weight;
    float s = 0.f;
    const long long stride = (long long)gridDim.x * blockDim.x;
    if (vec) {
        const float4* x4 = reinterpret_cast<const float4*>(x);
        float4* g4 = reinterpret_cast<float4*>(grad);
        for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n / 4; i += stride) {
            const float4 v = x4[i];
            s += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
            g4[i] = make_float4(k * v.x, k * v.y, k * v.z, k * v.w);
        }
    } else {
        for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += stride) {
            const float v = x[i];
            s += v * v;
            grad[i] = k * v;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    __shared__ float ss[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) ss[w] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0;
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) t += ss[i];
        atomicAdd(acc, t);
    }
}

__global__ void k_sumsq_loss(float weight, const double* __restrict__ acc, float* __restrict__ loss) {
    *loss = (float)(weight * *acc);
}

__global__ void k_add_inplace(long long n, float* __restrict__ dst, const float* __restrict__ src) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        dst[i] += src[i];
}

// 8-bit image values -> float32 in [0, 1] (k / 255, IEEE division); four
// bytes per thread and step
__global__ void k_u8_to_f32(long long n, const unsigned char* __restrict__ src, float* __restrict__ dst) {
    const long long n4 = n / 4;
    const uchar4* s4 = reinterpret_cast<const uchar4*>(src);
    float4* d4 = reinterpret_cast<float4*>(dst);
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n4; i += stride) {
        const uchar4 q = s4[i];
        d4[i] = make_float4((float)q.x / 255.f, (float)q.y / 255.f, (float)q.z / 255.f, (float)q.w / 255.f);
    }
    for (long long i = 4 * n4 + blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += stride)
        dst[i] = (float)src[i] / 255.f;
}

// Gaussian smoothing of images (Projects/CustomTFOperators/GaussianSmoothingGpu.py:12-37):
// a depthwise (2s+1)^2 convolution with the normalised outer product of a
// sampled normal density, zero padding ("SAME").  The kernel is separable: a
// CTA walks down a strip of rows, NC float columns per thread (a pixel row is
// W * Cn floats, its horizontal taps Cn floats apart), filters each row
// horizontally from shared memory (the next row's loads in flight) and keeps
// the last 2s+1 results of a column in registers for the vertical filter, so
// every input is read once but for the strips' halos, and no index is divided.
// Bound by HBM: 24 bytes per RGB pixel.  8 x 1024^2 RGB, s = 3: 59 us (3.4
// TB/s); 32 x 32 tiles in shared memory with a division per index took 321 us.
// Columns per thread: four while their registers leave eight CTAs per SM (s <=
// 3), two to s = 7, then one.
constexpr int kSmoothMax = 15;
constexpr int kSmoothBlock = 128;

struct SmoothTaps {
    float w[2 * kSmoothMax + 1];
};

template <int S>
constexpr int smooth_columns() { return S <= 3 ? 4 : S <= 7 ? 2 : 1; }

// CN: channels, or 0 to take them from Cn.  The n columns from `in` and `out` on
// are written; columns lo to hi (exclusive) belong to the image, whose rows have
// WC.
template <int S, int CN>
__global__ void __launch_bounds__(kSmoothBlock) k_smooth(int H, long long WC, int lo, int hi, int n, int Cn,
                                                         int rows_per_strip, SmoothTaps taps,
                                                         const float* __restrict__ in, float* __restrict__ out) {
    constexpr int T = kSmoothBlock, NC = smooth_columns<S>(), K = 2 * S + 1;
    static_assert(2 * kSmoothMax * 4 <= T, "one extra load per thread covers the halo");
    __shared__ float s_row[2][T * NC + 2 * S * 4];
    const int cn = CN ? CN : Cn, halo = S * cn, t = threadIdx.x;
    const int x0 = blockIdx.x * (T * NC), y0 = blockIdx.y * rows_per_strip;
    const int rows = min(rows_per_strip, H - y0) + 2 * S;
    const float* I = in + (long long)blockIdx.z * H * WC;
    float* O = out + (long long)blockIdx.z * H * WC;
    float next[NC + 1];
    auto fetch = [&](int r) {
        const int y = y0 - S + r;
        const bool ok = y >= 0 && y < H;
        const float* row = I + y * WC;
#pragma unroll
        for (int c = 0; c <= NC; ++c) {
            const int x = x0 - halo + t + c * T;
            next[c] = ok && x >= lo && x < hi && (c < NC || t < 2 * halo) ? row[x] : 0.f;
        }
    };
    fetch(0);
    float ring[NC][K];
    for (int r0 = 0; r0 < rows; r0 += K) {
#pragma unroll
        for (int u = 0; u < K; ++u) {
            const int r = r0 + u;
            if (r < rows) {  // CTA-uniform
                // the buffer was last read two rows ago, before the barrier between
                float* s = s_row[r & 1];
#pragma unroll
                for (int c = 0; c < NC; ++c) s[t + c * T] = next[c];
                if (t < 2 * halo) s[t + NC * T] = next[NC];
                __syncthreads();
                if (r + 1 < rows) fetch(r + 1);
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    float acc = 0.f;
#pragma unroll
                    for (int k = 0; k < K; ++k) acc += taps.w[k] * s[t + c * T + k * cn];
                    ring[c][u] = acc;
                }
                if (r >= 2 * S) {
                    float* row = O + (y0 + r - 2 * S) * WC + x0;
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        float acc = 0.f;
#pragma unroll
                        for (int k = 0; k < K; ++k) acc += taps.w[k] * ring[c][(u + 1 + k) % K];  // oldest row first
                        if (x0 + t + c * T < n) row[t + c * T] = acc;
                    }
                }
            }
        }
    }
}

// Columns of a launch: a row of an image may have more floats than 32 bits count.
constexpr long long kSmoothColumns = 1ll << 30;

template <int S>
hc_status launch_smooth(cudaStream_t s, int images, int H, int W, int Cn, const SmoothTaps& taps, const float* in,
                        float* out) {
    const long long WC = (long long)W * Cn;
    for (long long x = 0; x < WC; x += kSmoothColumns) {
        const int n = (int)std::min(kSmoothColumns, WC - x), gx = div_up(n, kSmoothBlock * smooth_columns<S>());
        const int lo = x > 0 ? -S * Cn : 0, hi = (int)std::min(WC - x, (long long)n + S * Cn);
        // 64-row strips; shorter ones while they leave SMs idle (their halos cost less than that)
        int rows = 64;
        while (rows > 8 && (long long)gx * div_up(H, rows) * images < 4 * 148) rows /= 2;
        while (div_up(H, rows) > 65535) rows *= 2;  // grid limit
        const dim3 grid(gx, div_up(H, rows), images);
        if (Cn == 3) k_smooth<S, 3><<<grid, kSmoothBlock, 0, s>>>(H, WC, lo, hi, n, Cn, rows, taps, in + x, out + x);
        else k_smooth<S, 0><<<grid, kSmoothBlock, 0, s>>>(H, WC, lo, hi, n, Cn, rows, taps, in + x, out + x);
        HC_CHECK_LAUNCH();
    }
    return HC_OK;
}

}  // namespace
}  // namespace hc

using namespace hc;

extern "C" hc_status hc_gaussian_smooth(void* stream, int32_t n_images, int32_t height, int32_t width,
                                        int32_t channels, int32_t size, float mean, float std, const float* image,
                                        float* out) {
    clear_error();
    HC_REQUIRE(n_images >= 0 && height > 0 && width > 0 && channels > 0 && channels <= 4, "bad sizes");
    HC_REQUIRE(size >= 0 && size <= kSmoothMax, "kernel size %d outside [0, %d]", size, kSmoothMax);
    HC_REQUIRE(image && out, "NULL pointer");
    HC_REQUIRE(image != out || size == 0 || std == 0.f, "in-place smoothing is not supported");
    cudaStream_t s = (cudaStream_t)stream;
    const size_t bytes = sizeof(float) * (size_t)n_images * height * width * channels;
    if (size == 0 || std == 0.f) {  // the reference returns the image unchanged
        if (image != out && bytes) HC_CUDA(cudaMemcpyAsync(out, image, bytes, cudaMemcpyDeviceToDevice, s));
        return HC_OK;
    }
    if (n_images == 0) return HC_OK;
    // normal density at -size..size, normalised so the 2-D kernel sums to one
    SmoothTaps t;
    double v[2 * kSmoothMax + 1], sum = 0.0;
    for (int k = 0; k <= 2 * size; ++k) {
        const double z = ((double)(k - size) - mean) / std;
        v[k] = exp(-0.5 * z * z);
        sum += v[k];
    }
    for (int k = 0; k <= 2 * size; ++k) t.w[k] = (float)(v[k] / sum);
    switch (size) {
#define HC_SMOOTH_CASE(S) \
    case S: return launch_smooth<S>(s, n_images, height, width, channels, t, image, out);
        HC_SMOOTH_CASE(1) HC_SMOOTH_CASE(2) HC_SMOOTH_CASE(3) HC_SMOOTH_CASE(4) HC_SMOOTH_CASE(5)
        HC_SMOOTH_CASE(6) HC_SMOOTH_CASE(7) HC_SMOOTH_CASE(8) HC_SMOOTH_CASE(9) HC_SMOOTH_CASE(10)
        HC_SMOOTH_CASE(11) HC_SMOOTH_CASE(12) HC_SMOOTH_CASE(13) HC_SMOOTH_CASE(14) HC_SMOOTH_CASE(15)
#undef HC_SMOOTH_CASE
    }
    return HC_OK;
}

extern "C" hc_status hc_sum_squares_loss(void* stream, int64_t n, const float* x, float weight, void* workspace,
                                         float* loss, float* grad) {
    clear_error();
    HC_REQUIRE(n >= 0, "n < 0");
    HC_REQUIRE(x && workspace && grad, "NULL input/output pointer");
    cudaStream_t s = (cudaStream_t)stream;
    double* acc = (double*)workspace;
    HC_CUDA(cudaMemsetAsync(acc, 0, sizeof(double), s));
    // grid-stride: as many CTAs as are resident at once, so that no partial
    // second wave runs after the rest
    const unsigned blocks = resident_grid(k_sumsq_fused, 256, n / 1024 + 1);
    const int vec = n % 4 == 0 && ((uintptr_t)x & 15) == 0 && ((uintptr_t)grad & 15) == 0;
    k_sumsq_fused<<<blocks, 256, 0, s>>>(n, x, weight, acc, grad, vec);
    HC_CHECK_LAUNCH();
    if (loss) {
        k_sumsq_loss<<<1, 1, 0, s>>>(weight, acc, loss);
        HC_CHECK_LAUNCH();
    }
    return HC_OK;
}

extern "C" hc_status hc_add_inplace(void* stream, int64_t n, float* dst, const float* src) {
    clear_error();
    HC_REQUIRE(n >= 0, "n < 0");
    HC_REQUIRE(dst && src, "NULL pointer");
    if (n == 0) return HC_OK;
    const long long blocks = n / 1024 + 1 < 148 * 8 ? n / 1024 + 1 : 148 * 8;
    k_add_inplace<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(n, dst, src);
    HC_CHECK_LAUNCH();
    return HC_OK;
}

extern "C" hc_status hc_image_u8_to_f32(void* stream, int64_t n, const uint8_t* src, float* dst) {
    clear_error();
    HC_REQUIRE(n >= 0, "n < 0");
    HC_REQUIRE(src && dst, "NULL pointer");
    HC_REQUIRE(((uintptr_t)src & 3) == 0 && ((uintptr_t)dst & 15) == 0,
               "src must be 4-byte and dst 16-byte aligned");
    if (n == 0) return HC_OK;
    const long long blocks = n / 4096 + 1 < 148 * 8 ? n / 4096 + 1 : 148 * 8;
    k_u8_to_f32<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(n, src, dst);
    HC_CHECK_LAUNCH();
    return HC_OK;
}

extern "C" hc_status hc_image_l1_loss_scratch(void* stream, int64_t n_pixels, const float* render_buffer,
                                              const float* target_image, const int32_t* face_buffer,
                                              const uint8_t* foreground_mask, void* workspace, uint8_t* scratch,
                                              float* loss, float* render_buffer_grad) {
    HC_REQUIRE(n_pixels <= 0 || scratch, "scratch is NULL");
    // 16-byte loads and stores; other addresses take the pair without scratch
    const uintptr_t at = (uintptr_t)render_buffer | (uintptr_t)target_image | (uintptr_t)face_buffer |
                         (uintptr_t)render_buffer_grad;
    if (n_pixels <= 0 || !render_buffer || !target_image || !face_buffer || !workspace || !render_buffer_grad ||
        (at & 15) != 0 || ((uintptr_t)scratch & 3) != 0)
        return hc_image_l1_loss(stream, n_pixels, render_buffer, target_image, face_buffer, foreground_mask, workspace,
                                loss, render_buffer_grad);
    clear_error();
    cudaStream_t s = (cudaStream_t)stream;
    L1Acc* acc = (L1Acc*)workspace;
    HC_CUDA(cudaMemsetAsync(acc, 0, sizeof(L1Acc), s));
    k_l1_signs<<<resident_grid(k_l1_signs, 256, n_pixels / 1024 + 1), 256, 0, s>>>(
        n_pixels, reinterpret_cast<const float4*>(render_buffer), reinterpret_cast<const float4*>(target_image),
        reinterpret_cast<const int4*>(face_buffer), foreground_mask, acc, scratch);
    HC_CHECK_LAUNCH();
    k_l1_from_signs<<<resident_grid(k_l1_from_signs, 256, n_pixels / 1024 + 1), 256, 0, s>>>(
        3 * n_pixels, scratch, acc, reinterpret_cast<float4*>(render_buffer_grad), loss);
    HC_CHECK_LAUNCH();
    return HC_OK;
}

extern "C" hc_status hc_image_l1_loss(void* stream, int64_t n_pixels, const float* render_buffer,
                                      const float* target_image, const int32_t* face_buffer,
                                      const uint8_t* foreground_mask, void* workspace, float* loss,
                                      float* render_buffer_grad) {
    clear_error();
    HC_REQUIRE(n_pixels >= 0, "n_pixels < 0");
    HC_REQUIRE(render_buffer && target_image && face_buffer && workspace && render_buffer_grad,
               "NULL input/output pointer");
    cudaStream_t s = (cudaStream_t)stream;
    L1Acc* acc = (L1Acc*)workspace;
    HC_CUDA(cudaMemsetAsync(acc, 0, sizeof(L1Acc), s));
    const int blocks = 148 * 8;
    k_l1_reduce<<<blocks, 256, 0, s>>>(n_pixels, render_buffer, target_image, face_buffer, foreground_mask, acc);
    HC_CHECK_LAUNCH();
    k_l1_grad<<<blocks, 256, 0, s>>>(n_pixels, render_buffer, target_image, face_buffer, foreground_mask, acc,
                                     render_buffer_grad, loss);
    HC_CHECK_LAUNCH();
    return HC_OK;
}
