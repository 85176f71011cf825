// A CUDA runtime on host memory, for tests of the engine's host side without a
// GPU: bh_engine.cu, compiled as C++, links against this file instead of the
// runtime and the kernels.  A stream is a queue whose operations run when
// something waits for them, so what a call leaves queued can be seen; copies of
// pageable memory are complete when they return, as the runtime's are.  Kernels
// do nothing but set the error words that a test asks for.
#include <cuda_runtime_api.h>

#include <atomic>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <map>
#include <mutex>

#include "../galaxy_b200/csrc/bh_internal.cuh"

namespace {

struct Stream {
    std::mutex mu;
    std::deque<std::function<void()>> ops;
    uint64_t issued = 0, executed = 0;
    void add(std::function<void()> op) {
        std::lock_guard<std::mutex> lk(mu);
        ops.push_back(std::move(op));
        ++issued;
    }
    void run(uint64_t upto) {
        std::lock_guard<std::mutex> lk(mu);
        while (executed < upto && !ops.empty()) {
            ops.front()();
            ops.pop_front();
            ++executed;
        }
    }
};
struct Event {
    Stream* stream = nullptr;
    uint64_t at = 0;
};

std::mutex g_mu;
std::map<const char*, size_t> g_pinned;  // cudaMallocHost blocks, and a test's arrays
bool g_capturing = false;
std::atomic<int> g_transfers{0};  // queued copies from or to host memory
int g_fail_after = -1;       // fallible calls until one fails (-1: none does)
uint32_t g_rebuild_err = 0;  // error bits that the next sorts set
uint32_t g_packed_err = 0;   // and the packed walks
uint32_t* g_step_err = nullptr;  // the error word of the steps captured last

Stream* of(cudaStream_t s) { return reinterpret_cast<Stream*>(s); }

bool pinned(const void* p) {
    std::lock_guard<std::mutex> lk(g_mu);
    auto it = g_pinned.upper_bound(static_cast<const char*>(p));
    if (it == g_pinned.begin()) return false;
    --it;
    return static_cast<const char*>(p) < it->first + it->second;
}

cudaError_t fallible() {
    std::lock_guard<std::mutex> lk(g_mu);
    return g_fail_after >= 0 && g_fail_after-- == 0 ? cudaErrorUnknown : cudaSuccess;
}

cudaError_t kernel(cudaStream_t s, std::function<void()> op = [] {}) {
    const cudaError_t e = fallible();
    if (e == cudaSuccess && !g_capturing) of(s)->add(std::move(op));
    return e;
}

}  // namespace

// -- controls of the tests ----------------------------------------------------
extern "C" {
void fake_reset() {
    g_fail_after = -1;
    g_rebuild_err = g_packed_err = 0;
    g_step_err = nullptr;
}
void fake_pin(const char* p, size_t n) { g_pinned[p] = n; }
void fake_unpin(const char* p) { g_pinned.erase(p); }
void fake_fail_after(int calls) { g_fail_after = calls; }
int fake_failed() { return g_fail_after == -1; }  // after fake_fail_after: whether it did
void fake_rebuild_error(uint32_t bits) { g_rebuild_err = bits; }
void fake_packed_error(uint32_t bits) { g_packed_err = bits; }
int fake_transfers() { return g_transfers; }

// -- the runtime ----------------------------------------------------------------
cudaError_t cudaDriverGetVersion(int* v) { return *v = 0, cudaSuccess; }
cudaError_t cudaRuntimeGetVersion(int* v) { return *v = 0, cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { return *n = 1, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) { return *p = {}, cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorName(cudaError_t) { return "fake"; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaMalloc(void** p, size_t n) { return *p = calloc(1, n), cudaSuccess; }
cudaError_t cudaFree(void* p) { return free(p), cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) {
    std::lock_guard<std::mutex> lk(g_mu);
    *p = calloc(1, n);
    g_pinned[static_cast<char*>(*p)] = n;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    std::lock_guard<std::mutex> lk(g_mu);
    g_pinned.erase(static_cast<char*>(p));
    return free(p), cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    *a = {};
    a->type = pinned(p) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) {
    return *p = reinterpret_cast<cudaMemPool_t>(new int), cudaSuccess;
}
cudaError_t cudaMemPoolDestroy(cudaMemPool_t p) {
    return delete reinterpret_cast<int*>(p), cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) {
    return *p = calloc(1, n), cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t s) {
    return of(s)->add([p] { free(p); }), cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    return *s = reinterpret_cast<cudaStream_t>(new Stream()), cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { return of(s)->run(~0ull), cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
    return *e = reinterpret_cast<cudaEvent_t>(new Event()), cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    return delete reinterpret_cast<Event*>(e), cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    if (g_capturing) return cudaSuccess;
    Event& ev = *reinterpret_cast<Event*>(e);
    std::lock_guard<std::mutex> lk(of(s)->mu);
    ev = Event{of(s), of(s)->issued};
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    Event& ev = *reinterpret_cast<Event*>(e);
    if (ev.stream) ev.stream->run(ev.at);
    return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    return *ms = 1.f, cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind kind,
                            cudaStream_t s) {
    const cudaError_t e = fallible();
    if (e != cudaSuccess) return e;
    ++g_transfers;
    of(s)->add([=] {
        memcpy(dst, src, n);
        --g_transfers;
    });
    if (kind != cudaMemcpyDeviceToDevice && !pinned(kind == cudaMemcpyHostToDevice ? src : dst))
        of(s)->run(~0ull);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t s) {
    return kernel(s, [=] { memset(p, v, n); });
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
    return g_capturing = true, cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
    return g_capturing = false, *g = nullptr, cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* g, cudaGraph_t, unsigned long long) {
    return *g = reinterpret_cast<cudaGraphExec_t>(1), cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t s) {
    return kernel(s, [] {
        if (g_step_err) *g_step_err |= g_rebuild_err;
    });
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
}  // extern "C"

// -- the kernels ------------------------------------------------------------------
namespace gbh {
bool small_sort(const BatchBuffers&) { return false; }
uint32_t probe_slices(uint32_t, uint32_t) { return 1; }
uint32_t conservation_blocks(uint32_t) { return 1; }
cudaError_t launch_integrate(const BatchBuffers&, int, cudaStream_t s) { return kernel(s); }
cudaError_t launch_morton(const BatchBuffers&, cudaStream_t s) { return kernel(s); }
cudaError_t launch_radix(const BatchBuffers& b, cudaStream_t s) {
    if (g_capturing) g_step_err = b.err;
    return kernel(s, [err = b.err] { *err |= g_rebuild_err; });
}
cudaError_t launch_sort_small(const BatchBuffers&, int, bool, cudaStream_t s) { return kernel(s); }
cudaError_t launch_count_scan(const BatchBuffers& b, cudaStream_t s) {
    // every position a cell of its own
    return kernel(s, [base = b.base, n = b.npos] {
        for (uint32_t p = 0; p <= n; ++p) base[p] = p;
    });
}
cudaError_t launch_aggregate(const BatchBuffers&, cudaStream_t s) { return kernel(s); }
cudaError_t launch_refresh_mac(const BatchBuffers&, uint32_t, cudaStream_t s) { return kernel(s); }
cudaError_t launch_wait_probe(uint32_t*, uint32_t*, long long, uint32_t*, cudaStream_t s) {
    return kernel(s);
}
cudaError_t launch_traverse(const BatchBuffers&, bool, bool, bool, bool, cudaStream_t s) {
    return kernel(s);
}
cudaError_t launch_export(const BatchBuffers&, uint32_t, GpuEntry*, GpuBody*, GpuCell*,
                          cudaStream_t s) {
    return kernel(s);
}
cudaError_t launch_traverse_packed(const BhSettings*, const GpuBody*, const GpuEntry*,
                                   const GpuCell*, uint32_t, uint32_t, float4*, uint32_t* err,
                                   cudaStream_t s) {
    return kernel(s, [err] { *err |= g_packed_err; });
}
cudaError_t launch_direct_probes(const GpuEvolveState*, uint32_t, const uint32_t*, uint32_t,
                                 double, double, double*, cudaStream_t s) {
    return kernel(s);
}
cudaError_t launch_traverse_f64(const BatchBuffers&, uint32_t, uint32_t, double, double, double,
                                double*, double*, unsigned long long*, cudaStream_t s) {
    return kernel(s);
}
cudaError_t launch_conservation(const GpuEvolveState*, const float*, uint32_t, double*, uint32_t,
                                double*, cudaStream_t s) {
    return kernel(s);
}
cudaError_t launch_check_records(const void*, int, uint32_t, uint32_t*, cudaStream_t s) {
    return kernel(s);
}
}  // namespace gbh
