// Error reporting for the C ABI.
#include <atomic>

#include "hc_common.cuh"

#include <map>
#include <mutex>
#include <tuple>

namespace hc {

static thread_local std::string g_last_error;

void set_error(const char* fmt, ...) {
    char buf[1024];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    g_last_error = buf;
}

void clear_error() { g_last_error.clear(); }

static std::atomic<long long> g_launches{0};
void count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }

int resident_ctas(const void* kernel, int threads) {
    static std::mutex mu;
    static std::map<std::tuple<const void*, int, int>, int> known;  // a few kernels per device
    int dev = 0, sms = 0, per_sm = 0;
    std::lock_guard<std::mutex> lock(mu);
    bool ok = cudaGetDevice(&dev) == cudaSuccess;
    const auto it = ok ? known.find({kernel, threads, dev}) : known.end();
    if (it != known.end()) return it->second;
    ok = ok && cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && sms > 0 &&
         cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, 0) == cudaSuccess && per_sm > 0;
    if (!ok) {  // a guess for this call alone; the error is not the launch's
        cudaGetLastError();
        return 148;
    }
    return known[{kernel, threads, dev}] = sms * per_sm;
}

__global__ void k_fill(FillRuns runs) {
    fill_runs(runs, blockIdx.x * (long long)blockDim.x + threadIdx.x, gridDim.x * (long long)blockDim.x);
}

hc_status fill(const FillRuns& runs, cudaStream_t s) {
    k_fill<<<runs.blocks(256), 256, 0, s>>>(runs);
    HC_CHECK_LAUNCH();
    return HC_OK;
}

}  // namespace hc

extern "C" const char* hc_last_error(void) { return hc::g_last_error.c_str(); }
extern "C" const char* hc_version(void) { return "hc-b200 0.1 (sm_100a)"; }
extern "C" int64_t hc_kernel_launches(void) { return hc::g_launches.load(std::memory_order_relaxed); }
