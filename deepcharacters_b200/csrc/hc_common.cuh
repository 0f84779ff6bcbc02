// Runtime plumbing shared by the C-ABI entry points: status codes, the
// per-thread error message, CUDA error checks and a grow-only device buffer.
#pragma once

#include <cuda_runtime.h>
#include <stdarg.h>
#include <stdint.h>
#include <stdio.h>

#include <string>

#include "../../include/hc.h"

namespace hc {

void set_error(const char* fmt, ...);
void clear_error();
// process-wide count of kernel launches issued by this library
void count_launch();

#define HC_FAIL(code, ...)            \
    do {                              \
        ::hc::set_error(__VA_ARGS__); \
        return (code);                \
    } while (0)

#define HC_CUDA(call)                                                                       \
    do {                                                                                    \
        cudaError_t e_ = (call);                                                            \
        if (e_ != cudaSuccess)                                                              \
            HC_FAIL(HC_ERR_CUDA, "%s:%d %s: %s", __FILE__, __LINE__, #call, cudaGetErrorString(e_)); \
    } while (0)

#define HC_CHECK_LAUNCH()         \
    do {                          \
        ::hc::count_launch();     \
        HC_CUDA(cudaGetLastError()); \
    } while (0)

#define HC_REQUIRE(cond, ...)                                \
    do {                                                     \
        if (!(cond)) HC_FAIL(HC_ERR_INVALID, __VA_ARGS__);   \
    } while (0)

#define HC_TRY(expr)                    \
    do {                                \
        hc_status s_ = (expr);          \
        if (s_ != HC_OK) return s_;     \
    } while (0)

// Device allocation that only grows; freed by the owner's destructor.
struct DevBuf {
    void* ptr = nullptr;
    size_t bytes = 0;
    hc_status ensure(size_t need) {
        if (need <= bytes) return HC_OK;
        if (ptr) cudaFree(ptr);
        ptr = nullptr;
        bytes = 0;
        if (need == 0) return HC_OK;
        cudaError_t e = cudaMalloc(&ptr, need);
        if (e != cudaSuccess) {
            ptr = nullptr;
            cudaGetLastError();  // reported here, not by the next launch's check
            HC_FAIL(HC_ERR_ALLOC, "cudaMalloc(%zu) failed: %s", need, cudaGetErrorString(e));
        }
        bytes = need;
        return HC_OK;
    }
    void release() {
        if (ptr) cudaFree(ptr);
        ptr = nullptr;
        bytes = 0;
    }
    template <class T>
    T* as() const { return reinterpret_cast<T*>(ptr); }
};

// One of several arrays in an allocation.
struct DevPart {
    void* ptr = nullptr;
    template <class T>
    T* as() const { return reinterpret_cast<T*>(ptr); }
};

// Scratch that a call is faster with and can do without: there is no room where
// memory is short, where a capture would have to allocate it, and where growing it
// would free what a captured graph addresses.
struct SpareBuf : DevBuf {
    bool captured = false;  // a graph holds its address: it keeps its size
    size_t refused = ~(size_t)0;  // there was no memory for this size
    int patience = 0;             // calls until it is asked for again (a failed attempt costs more than the scratch gains)
    bool room(size_t need, cudaStreamCaptureStatus capture) {
        const bool recording = capture != cudaStreamCaptureStatusNone;
        if (bytes < need) {
            if (captured || recording || (need >= refused && patience-- > 0)) return false;
            if (ensure(need) != HC_OK) {
                clear_error();
                refused = need;
                patience = 1000;
                return false;
            }
            refused = ~(size_t)0;
        }
        captured = captured || recording;
        return true;
    }
};

template <class T>
hc_status upload(DevBuf& b, const T* host, size_t count) {
    HC_TRY(b.ensure(count * sizeof(T)));
    if (count) HC_CUDA(cudaMemcpy(b.ptr, host, count * sizeof(T), cudaMemcpyHostToDevice));
    return HC_OK;
}

// CTAs of a kernel that are resident on the current device at once (SMs x CTAs
// per SM without dynamic shared memory); looked up once per kernel, block size
// and device
int resident_ctas(const void* kernel, int threads);

// grid of a persistent kernel: as many CTAs as are resident at once (a second
// partial wave would run its work after everything else), never more than the
// work items
template <typename K>
unsigned resident_grid(K kernel, int threads, long long items) {
    const long long g = resident_ctas(reinterpret_cast<const void*>(kernel), threads);
    return (unsigned)(items < 1 ? 1 : items < g ? items : g);
}

inline int div_up(long long a, long long b) { return (int)((a + b - 1) / b); }

// Device ranges to fill with a byte each, by one launch or by spare blocks of a
// kernel that is launched anyway: a memset of its own costs a launch (0.8 to 1.4
// us of device time and its gap) for a few bytes.
struct FillRuns {
    static constexpr int kMost = 6;
    char* p[kMost];
    long long n[kMost];
    unsigned word[kMost];  // the byte, four times
    int count = 0;
    void add(void* ptr, size_t bytes, unsigned char value = 0) {
        p[count] = static_cast<char*>(ptr);
        n[count] = (long long)bytes;
        word[count++] = 0x01010101u * value;
    }
    // blocks of `threads` that fill with four 16-byte stores a thread, at most a
    // few waves (the loop strides over the rest)
    unsigned blocks(int threads) const {
        long long b = 0;
        for (int i = 0; i < count; ++i) b += n[i];
        b = (b / 64 + threads - 1) / threads;
        return (unsigned)(b < 1 ? 1 : b < 148 * 16 ? b : 148 * 16);
    }
};

// thread t of nt fills its share of the ranges (any alignment, any size)
__device__ __forceinline__ void fill_runs(const FillRuns& r, long long t, long long nt) {
#pragma unroll
    for (int i = 0; i < FillRuns::kMost; ++i) {
        if (i >= r.count) break;
        char* p = r.p[i];
        const long long off = (long long)(-(uintptr_t)p & 15), head = off < r.n[i] ? off : r.n[i];
        const long long body = (r.n[i] - head) >> 4, tail = head + (body << 4);
        uint4* q = reinterpret_cast<uint4*>(p + head);
        const uint4 w = make_uint4(r.word[i], r.word[i], r.word[i], r.word[i]);
        for (long long k = t; k < body; k += nt) q[k] = w;
        for (long long k = t; k < head; k += nt) p[k] = (char)r.word[i];
        for (long long k = tail + t; k < r.n[i]; k += nt) p[k] = (char)r.word[i];
    }
}

hc_status fill(const FillRuns& runs, cudaStream_t s);

}  // namespace hc
