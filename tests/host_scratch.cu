// Host checks of the library's buffers, against a fake of the CUDA runtime calls
// that they make: run with the name of a check, exit code 0 when it holds.
#include <cstdlib>
#include <cstring>
#include <map>

#include "../deepcharacters_b200/csrc/renderer.cuh"

namespace fake {
size_t room = ~(size_t)0;  // the largest allocation that succeeds
int mallocs = 0, frees = 0;
std::map<void*, size_t> live;
cudaError_t last = cudaSuccess;
cudaStreamCaptureMode mode = cudaStreamCaptureModeGlobal;
bool recording = false;  // allocations and frees are refused unless the mode is relaxed
bool refused() { return recording && mode != cudaStreamCaptureModeRelaxed; }
cudaError_t fail(cudaError_t e) { return last = e; }
int device = 0, queries = 0;
bool occupancy_fails = false;
}  // namespace fake

#ifndef __CUDA_ARCH__
extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) {
    ++fake::mallocs;
    if (fake::refused()) return fake::fail(cudaErrorStreamCaptureUnsupported);
    if (n > fake::room) return fake::fail(cudaErrorMemoryAllocation);
    fake::live[*p = std::malloc(16)] = n;  // never freed: each has an address of its own
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    ++fake::frees;
    if (fake::refused()) return fake::fail(cudaErrorStreamCaptureUnsupported);
    return fake::live.erase(p) ? cudaSuccess : fake::fail(cudaErrorInvalidValue);
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = fake::last;
    fake::last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode* m) {
    std::swap(*m, fake::mode);
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
    *d = fake::device;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) {
    *v = 10;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int threads, size_t) {
    ++fake::queries;
    if (fake::occupancy_fails) return fake::fail(cudaErrorInvalidValue);
    *n = 1024 / threads + fake::device;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return cudaSuccess; }
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, struct CUstream_st*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
cudaError_t cudaMemcpy(void*, const void*, size_t, cudaMemcpyKind) { return cudaSuccess; }
void** __cudaRegisterFatBinary(void*) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
char __cudaInitModule(void**) { return 0; }
}
#endif

using namespace hc;

#define CHECK(c)                                                  \
    do {                                                          \
        if (!(c)) {                                               \
            fprintf(stderr, "line %d: %s\n", __LINE__, #c);       \
            return 1;                                             \
        }                                                         \
    } while (0)

const cudaStreamCaptureStatus kEager = cudaStreamCaptureStatusNone, kRecord = cudaStreamCaptureStatusActive;

// A call at a size, as the UV maps make it; the table it used, NULL where it failed.
static UvTable* uv_call(UvTables& t, int size, cudaStreamCaptureStatus capture, bool* built = nullptr) {
    fake::recording = capture != kEager;
    UvTable* k = nullptr;
    const hc_status st = t.get(size, size, capture, &k);
    fake::recording = false;
    if (st != HC_OK) return nullptr;
    if (built) *built = !k->valid;
    if (!k->valid) k->valid = capture == kEager;
    return k;
}

// a table that a graph holds is neither replaced nor built again for another size
static int uv_held() {
    UvTables t;
    bool built = false;
    CHECK(uv_call(t, 37, kEager, &built) && built);
    void* at = uv_call(t, 37, kRecord, &built)->buf.ptr;
    CHECK(!built && fake::mallocs == 1);
    const UvTable* big = uv_call(t, 64, kEager, &built);
    CHECK(big && built && big->buf.ptr != at && fake::frees == 0);
    const UvTable* small = uv_call(t, 16, kEager, &built);  // in the place of the 64^2 table
    CHECK(small && built && small->buf.ptr != at && t.tables.size() == 2);
    const UvTable* again = uv_call(t, 37, kEager, &built);
    CHECK(again->buf.ptr == at && !built && again->th == 37 && fake::live.count(at));
    return 0;
}

// a table whose build was only recorded does not count as built
static int uv_recorded() {
    UvTables t;
    bool built = false;
    CHECK(uv_call(t, 64, kEager));
    void* at = uv_call(t, 37, kRecord, &built)->buf.ptr;  // fits, and is built at each replay
    CHECK(built && fake::mallocs == 1);
    CHECK(uv_call(t, 64, kEager, &built)->buf.ptr != at && built);
    CHECK(uv_call(t, 37, kEager, &built)->buf.ptr == at && built);
    CHECK(uv_call(t, 37, kEager, &built)->buf.ptr == at && !built);
    // a second graph of the size shares the table; one of another size that only a held
    // table has room for gets its own
    CHECK(uv_call(t, 37, kRecord)->buf.ptr == at);
    CHECK(uv_call(t, 64, kRecord, &built)->buf.ptr != at && !built);
    const size_t n = t.tables.size();
    const UvTable* k = uv_call(t, 20, kRecord, &built);
    CHECK(k && built && k->buf.ptr != at && t.tables.size() == n + 1 && fake::mode == cudaStreamCaptureModeGlobal);
    CHECK(!uv_call(t, 1024, kRecord));  // no table of that size was ever made: refused
    return 0;
}

// after a failed allocation no size is taken for built
static int uv_no_memory() {
    UvTables t;
    bool built = false;
    CHECK(uv_call(t, 37, kEager));
    fake::room = 1 << 16;
    CHECK(!uv_call(t, 64, kEager));
    const UvTable* k = uv_call(t, 37, kEager, &built);
    CHECK(k && built && k->buf.ptr && k->buf.bytes >= 20u * 37 * 37);
    return 0;
}

// a vertex's entry names its place in the face and the others in the face's order
static int fan_entries() {
    const int face[5][3] = {{4, 7, 9}, {7, 4, 9}, {9, 7, 4}, {4, 4, 9}, {9, 4, 4}};  // the last two degenerate
    for (const auto& f : face)
        for (int v : {4, 7, 9}) {
            const int place = v == f[0] ? 0 : v == f[1] ? 1 : v == f[2] ? 2 : -1;
            if (place < 0) continue;
            const int2 e = fan_entry(v, f[0], f[1], f[2]);
            CHECK((unsigned)e.y >> 30 == (unsigned)place && e.x == f[place == 0 ? 1 : 0] &&
                  (e.y & 0x3fffffff) == f[place == 2 ? 1 : 2]);
        }
    return 0;
}

// spare scratch that a graph holds is neither replaced nor grown
static int spare_held() {
    SpareBuf b;
    CHECK(!b.room(100, kRecord) && !b.captured && b.room(100, kEager) && b.room(300, kEager));
    void* at = b.ptr;
    CHECK(b.room(200, kRecord) && b.captured);
    const int mallocs = fake::mallocs, frees = fake::frees;
    CHECK(!b.room(400, kEager) && !b.room(400, kRecord) && b.room(300, kEager));
    CHECK(b.ptr == at && b.bytes == 300 && fake::mallocs == mallocs && fake::frees == frees && fake::live.count(at));
    return 0;
}

// where memory is short the allocation is not tried again in every call
static int spare_no_memory() {
    SpareBuf b;
    CHECK(b.room(100, kEager));
    fake::room = 1000;
    for (int k = 0; k < 500; ++k) CHECK(!b.room(5000, kEager));
    CHECK(fake::mallocs == 2 && fake::last == cudaSuccess);
    CHECK(b.room(900, kEager) && b.bytes == 900);
    fake::room = 10000;
    bool found = false;
    for (int k = 0; k < 1000; ++k) found = found || b.room(5000, kEager);
    CHECK(found && b.bytes == 5000 && fake::mallocs == 4);
    return 0;
}

// a failed allocation is reported once, by the call that needed it
static int failed_allocation() {
    DevBuf b;
    CHECK(b.ensure(100) == HC_OK);
    fake::room = 1000;
    CHECK(b.ensure(2000) == HC_ERR_ALLOC && fake::last == cudaSuccess && !b.ptr && b.bytes == 0);
    CHECK(b.ensure(500) == HC_OK && b.bytes == 500);
    return 0;
}

// the resident CTAs are those of the kernel, the block size and the device; a failed
// query is neither kept nor left for the next launch to report
static int resident() {
    const void *a = &fake::room, *b = &fake::last;
    CHECK(resident_ctas(a, 256) == 40 && resident_ctas(a, 64) == 160 && resident_ctas(a, 256) == 40);
    CHECK(fake::queries == 2);
    fake::device = 1;
    CHECK(resident_ctas(a, 256) == 50 && resident_ctas(a, 64) == 170);
    fake::occupancy_fails = true;
    CHECK(resident_ctas(b, 256) > 0 && fake::last == cudaSuccess);
    fake::occupancy_fails = false;
    CHECK(resident_ctas(b, 256) == 50);
    return 0;
}

int main(int argc, char** argv) {
    const std::map<std::string, int (*)()> checks = {
        {"uv_held", uv_held},
        {"uv_recorded", uv_recorded},
        {"uv_no_memory", uv_no_memory},
        {"fan_entries", fan_entries},
        {"resident", resident},
        {"spare_held", spare_held},
        {"spare_no_memory", spare_no_memory},
        {"failed_allocation", failed_allocation},
    };
    const auto it = checks.find(argc > 1 ? argv[1] : "");
    return it == checks.end() ? 2 : it->second();
}
