// SPDX-License-Identifier: Apache-2.0
//
// Host runtime of the B200 Barnes-Hut engine and the C ABI of galaxy_bh.h.
//
// A Batch lays one or more simulations out in a shared "position space":
// simulation s owns positions [off_s, off_s + n_s), off_s a multiple of 32,
// so a warp never straddles two simulations.  Radix tiles (4096 keys) never
// straddle simulations either.  Per-rebuild scratch (keys, sorted bodies,
// cells, control block) is one device arena carved at batch creation and
// sized for the worst case, so no step ever allocates.  The plain API
// (tree_create / rebuild / force) is a batch of one.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <memory>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "bh_internal.cuh"

using namespace gbh;

// ------------------------------------------------------------------ errors --

static thread_local std::string g_last_error;

static int set_error(int status, const char* fmt, ...) {
    char buf[1024];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    g_last_error = buf;
    return status;
}

static int cuda_fail(cudaError_t e, const char* what) {
    cudaGetLastError();
    return set_error(e == cudaErrorMemoryAllocation ? BH_OOM : BH_CUDA_ERROR, "%s: %s (%s)", what,
                     cudaGetErrorName(e), cudaGetErrorString(e));
}

#define CK(expr, what)                                  \
    do {                                                \
        cudaError_t _e = (expr);                        \
        if (_e != cudaSuccess) return cuda_fail(_e, what); \
    } while (0)

int gbh::set_error_message(int status, const char* message) {
    return set_error(status, "%s", message);
}

extern "C" size_t galaxy_bh_last_error(char* buf, size_t len) {
    if (buf && len) {
        size_t n = std::min(len - 1, g_last_error.size());
        memcpy(buf, g_last_error.data(), n);
        buf[n] = 0;
    }
    return g_last_error.size();
}

extern "C" uint32_t galaxy_bh_abi_version(void) { return GALAXY_BH_ABI_VERSION; }

// ------------------------------------------------------------ host copies --

// Copies between device memory and a caller's pageable arrays, through pinned
// slots and with a few threads: the driver's own staging is one thread that
// faults in the caller's pages one by one.  Each thread takes every W-th chunk
// and has two slots, so its memcpy of one chunk runs beside the transfer of the
// next: read-back of 2^20 states 7.6 -> 3.3 ms, of 2^22 27.8 -> 13.0, upload of
// 2^22 12 -> 5.3.  The slots (4 MB) belong to the device handle and are made by
// its first copy that uses them (about 8 ms, once).  Arrays that are pinned
// already are copied as they are, and so are those below 16 MB: from 4 to 8 MB
// the threads cost up to a fifth more than they save, at 12 MB 10 % less, and a
// handle that moves no more than that need not pay for the slots.  Two host
// threads that copy their own states through one handle take the slots in turn.
class HostCopies {
public:
    // Returns once a device-to-host copy is complete; a host-to-device one may
    // still be running on the stream, but its source can be reused.
    cudaError_t run(void* dst, const void* src, size_t bytes, bool to_host, cudaStream_t stream,
                    int ordinal) {
        const void* host = to_host ? dst : src;
        cudaPointerAttributes at{};
        const bool pageable = cudaPointerGetAttributes(&at, host) != cudaSuccess ||
                              at.type == cudaMemoryTypeUnregistered;
        cudaGetLastError();
        const bool staged = pageable && bytes >= kStagedBytes;
        std::unique_lock<std::mutex> slots(in_use_, std::defer_lock);
        if (staged) slots.lock();
        if (!staged || !ready())
            return cudaMemcpyAsync(dst, src, bytes,
                                   to_host ? cudaMemcpyDeviceToHost : cudaMemcpyHostToDevice, stream);
        const size_t chunks = (bytes + kChunk - 1) / kChunk;
        const int workers = (int)std::min<size_t>(kWorkers, chunks);
        cudaError_t result[kWorkers] = {};
        auto work = [&](int w) {
            result[w] = cudaSetDevice(ordinal);
            if (result[w] == cudaSuccess)
                result[w] = to_host ? down(w, workers, (char*)dst, (const char*)src, bytes, stream)
                                    : up(w, workers, (char*)dst, (const char*)src, bytes, stream);
        };
        std::thread threads[kWorkers];
        for (int w = 1; w < workers; ++w) {
            try {
                threads[w] = std::thread(work, w);
            } catch (...) {  // no thread to be had: its share is done here
                work(w);
            }
        }
        work(0);
        cudaError_t e = result[0];
        for (int w = 1; w < workers; ++w) {
            if (threads[w].joinable()) threads[w].join();
            if (e == cudaSuccess) e = result[w];
        }
        return e;
    }

    void release() {
        for (auto& s : slots_)
            if (s.done) cudaEventDestroy(s.done);
        if (pinned_) cudaFreeHost(pinned_);
        pinned_ = nullptr;
        for (auto& s : slots_) s = Slot();
    }

private:
    static constexpr size_t kChunk = 512u << 10, kStagedBytes = 16u << 20;
    static constexpr int kWorkers = 4;
    struct Slot {
        char* at = nullptr;
        cudaEvent_t done = nullptr;
        bool used = false;
    };

    bool ready() {
        if (pinned_) return true;
        if (cudaMallocHost((void**)&pinned_, kChunk * 2 * kWorkers) != cudaSuccess) {
            cudaGetLastError();
            pinned_ = nullptr;
            return false;
        }
        for (int k = 0; k < 2 * kWorkers; ++k) {
            slots_[k].at = pinned_ + kChunk * k;
            if (cudaEventCreateWithFlags(&slots_[k].done, cudaEventDisableTiming) != cudaSuccess) {
                cudaGetLastError();
                release();
                return false;
            }
        }
        return true;
    }

    cudaError_t down(int w, int workers, char* dst, const char* src, size_t bytes,
                     cudaStream_t stream) {
        size_t pending = bytes;  // offset of the chunk in the other slot
        int k = 0;
        auto finish = [&](int slot, size_t at) -> cudaError_t {
            const cudaError_t e = cudaEventSynchronize(slots_[slot].done);
            if (e == cudaSuccess)
                memcpy(dst + at, slots_[slot].at, std::min(kChunk, bytes - at));
            return e;
        };
        for (size_t at = (size_t)w * kChunk; at < bytes; at += workers * kChunk, k ^= 1) {
            Slot& s = slots_[2 * w + k];
            cudaError_t e = cudaMemcpyAsync(s.at, src + at, std::min(kChunk, bytes - at),
                                            cudaMemcpyDeviceToHost, stream);
            if (e == cudaSuccess) e = cudaEventRecord(s.done, stream);
            if (e == cudaSuccess && pending < bytes) e = finish(2 * w + (k ^ 1), pending);
            if (e != cudaSuccess) return e;
            s.used = false;  // waited for below or in the next turn
            pending = at;
        }
        return pending < bytes ? finish(2 * w + (k ^ 1), pending) : cudaSuccess;
    }

    cudaError_t up(int w, int workers, char* dst, const char* src, size_t bytes,
                   cudaStream_t stream) {
        int k = 0;
        for (size_t at = (size_t)w * kChunk; at < bytes; at += workers * kChunk, k ^= 1) {
            Slot& s = slots_[2 * w + k];
            cudaError_t e = s.used ? cudaEventSynchronize(s.done) : cudaSuccess;
            if (e != cudaSuccess) return e;
            const size_t size = std::min(kChunk, bytes - at);
            memcpy(s.at, src + at, size);
            e = cudaMemcpyAsync(dst + at, s.at, size, cudaMemcpyHostToDevice, stream);
            if (e == cudaSuccess) e = cudaEventRecord(s.done, stream);
            if (e != cudaSuccess) return e;
            s.used = true;
        }
        return cudaSuccess;
    }

    std::mutex in_use_;  // one copy at a time has the slots
    char* pinned_ = nullptr;
    Slot slots_[2 * kWorkers];
};

// ------------------------------------------------------------------ device --

struct bh_device {
    int ordinal = 0;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev[8] = {};
    cudaDeviceProp prop{};
    int refs = 0;         // live states, trees and batches on this device
    bool closed = false;  // galaxy_bh_device_close was called
    // Stream-ordered pool of the per-state buffers and the batch / tree
    // arenas.  It keeps released memory for reuse (trimmed only when an
    // allocation runs short): cudaFree synchronizes the whole device and
    // unmaps pages, which cost a serving loop seconds per burst of finished
    // requests and would stall it on its stager's work.
    cudaMemPool_t pool = nullptr;
    // Blocks above kSmallBlock that single calls take for their own length
    // (PoolBlock): it keeps at most kScratchKept, an export of 2^22 bodies takes 660
    // MB once.  Smaller ones come from `pool`, which mostly has room: a handle's
    // first few probes would take 300 us longer from a pool that has none yet.
    cudaMemPool_t scratch = nullptr;
    HostCopies copies;
};
constexpr uint64_t kSmallBlock = 32ull << 20, kScratchKept = 256ull << 20;

// Memory from one of the handle's pools; when it runs short, what they keep unused
// is given back and tried again.
static cudaError_t pool_alloc(bh_device* dev, cudaMemPool_t pool, void** at, size_t bytes) {
    cudaError_t e = cudaMallocFromPoolAsync(at, bytes, pool, dev->stream);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        cudaStreamSynchronize(dev->stream);
        cudaMemPoolTrimTo(dev->pool, 0);
        cudaMemPoolTrimTo(dev->scratch, 0);
        e = cudaMallocFromPoolAsync(at, bytes, pool, dev->stream);
    }
    if (e != cudaSuccess) *at = nullptr;
    return e;
}

static cudaError_t copy_down(bh_device* dev, void* host, const void* device, size_t bytes) {
    return dev->copies.run(host, device, bytes, true, dev->stream, dev->ordinal);
}
static cudaError_t copy_up(bh_device* dev, void* device, const void* host, size_t bytes) {
    return dev->copies.run(device, host, bytes, false, dev->stream, dev->ordinal);
}

// Device memory of one call from the handle's pools (no device-wide
// synchronisation, as cudaMalloc and cudaFree have), given back in stream order.
// A call that returns before wait() has ended well (an error on the way) waits
// here: what it has queued may still read or write the caller's arrays.
struct PoolBlock {
    bh_device* dev;
    char* at = nullptr;
    bool idle = false;  // nothing of the call is queued any more
    bool large = false;  // more than the pool keeps: it gives memory back when waited for
    explicit PoolBlock(bh_device* d) : dev(d) {}
    PoolBlock(const PoolBlock&) = delete;
    PoolBlock& operator=(const PoolBlock&) = delete;
    cudaError_t get(size_t bytes) {
        large = bytes > kScratchKept;
        return pool_alloc(dev, bytes > kSmallBlock ? dev->scratch : dev->pool, (void**)&at, bytes);
    }
    cudaError_t wait() {
        const cudaError_t e = cudaStreamSynchronize(dev->stream);
        idle = e == cudaSuccess;
        return e;
    }
    ~PoolBlock() {
        if (!at) return;
        cudaFreeAsync(at, dev->stream);
        if (!idle || large) cudaStreamSynchronize(dev->stream);
    }
};

static void device_free(bh_device* dev) {
    cudaSetDevice(dev->ordinal);
    cudaStreamSynchronize(dev->stream);
    dev->copies.release();
    if (dev->pool) cudaMemPoolDestroy(dev->pool);
    if (dev->scratch) cudaMemPoolDestroy(dev->scratch);
    for (auto& ev : dev->ev) cudaEventDestroy(ev);
    cudaStreamDestroy(dev->stream);
    delete dev;
}

static void device_ref(bh_device* dev) { ++dev->refs; }

// Drops one handle's reference; frees a closed device with no handles left.
static void device_unref(bh_device* dev) {
    if (!dev) return;
    if (--dev->refs == 0 && dev->closed) device_free(dev);
}

static int enter(bh_device* dev) {
    if (!dev) return set_error(BH_INVALID_ARG, "null device handle");
    if (dev->closed) return set_error(BH_INVALID_ARG, "device handle is closed");
    CK(cudaSetDevice(dev->ordinal), "cudaSetDevice");
    return BH_OK;
}

extern "C" int galaxy_bh_device_open(int ordinal, bh_device** out) {
    if (!out) return set_error(BH_INVALID_ARG, "null output pointer");
    *out = nullptr;
    int count = 0;
    cudaError_t e = cudaGetDeviceCount(&count);
    if (e != cudaSuccess || count == 0) {
        cudaGetLastError();
        return set_error(BH_NO_DEVICE, "No CUDA device is available (%s)",
                         e == cudaSuccess ? "0 devices" : cudaGetErrorName(e));
    }
    if (ordinal < 0 || ordinal >= count)
        return set_error(BH_NO_DEVICE, "CUDA device ordinal %d out of range (0..%d)", ordinal,
                         count - 1);
    bh_device* d = new bh_device();
    d->ordinal = ordinal;
    cudaMemPoolProps pool_props{};
    pool_props.allocType = cudaMemAllocationTypePinned;
    pool_props.location.type = cudaMemLocationTypeDevice;
    pool_props.location.id = ordinal;
    const uint64_t keep = ~0ull, scratch_keep = kScratchKept;
    if ((e = cudaSetDevice(ordinal)) != cudaSuccess ||
        (e = cudaGetDeviceProperties(&d->prop, ordinal)) != cudaSuccess ||
        (e = cudaStreamCreateWithFlags(&d->stream, cudaStreamNonBlocking)) != cudaSuccess ||
        (e = cudaMemPoolCreate(&d->pool, &pool_props)) != cudaSuccess ||
        (e = cudaMemPoolSetAttribute(d->pool, cudaMemPoolAttrReleaseThreshold,
                                     (void*)&keep)) != cudaSuccess ||
        (e = cudaMemPoolCreate(&d->scratch, &pool_props)) != cudaSuccess ||
        (e = cudaMemPoolSetAttribute(d->scratch, cudaMemPoolAttrReleaseThreshold,
                                     (void*)&scratch_keep)) != cudaSuccess) {
        if (d->pool) cudaMemPoolDestroy(d->pool);
        if (d->scratch) cudaMemPoolDestroy(d->scratch);
        if (d->stream) cudaStreamDestroy(d->stream);
        delete d;
        return cuda_fail(e, "device open");
    }
    for (auto& ev : d->ev) cudaEventCreate(&ev);
    *out = d;
    return BH_OK;
}

extern "C" int galaxy_bh_device_close(bh_device* dev) {
    if (!dev || dev->closed) return BH_OK;
    dev->closed = true;
    if (dev->refs == 0) device_free(dev);
    return BH_OK;
}

extern "C" int galaxy_bh_device_info(bh_device* dev, char* buf, size_t len) {
    int rc = enter(dev);
    if (rc) return rc;
    int rt = 0, drv = 0;
    cudaRuntimeGetVersion(&rt);
    cudaDriverGetVersion(&drv);
    char tmp[768];
    snprintf(tmp, sizeof tmp,
             "{\"index\": %d, \"name\": \"%s\", \"backend\": \"CUDA\", \"device_type\": "
             "\"DiscreteGpu\", \"compute_capability\": \"%d.%d\", \"sm_count\": %d, "
             "\"memory_bytes\": %zu, \"cuda_runtime\": %d, \"cuda_driver\": %d, "
             "\"software\": false}",
             dev->ordinal, dev->prop.name, dev->prop.major, dev->prop.minor,
             dev->prop.multiProcessorCount, (size_t)dev->prop.totalGlobalMem, rt, drv);
    if (buf && len) {
        strncpy(buf, tmp, len - 1);
        buf[len - 1] = 0;
    }
    return BH_OK;
}

extern "C" int galaxy_bh_device_stream(bh_device* dev, void** stream) {
    if (!dev || !stream) return set_error(BH_INVALID_ARG, "null argument");
    *stream = (void*)dev->stream;
    return BH_OK;
}

// ------------------------------------------------------------ config -------

static int validate_config(const bh_config* c) {
    if (!c) return set_error(BH_INVALID_ARG, "null config");
    // nbody/src/lib.rs:48-66
    if (!std::isfinite(c->theta) || c->theta < 0.0)
        return set_error(BH_INVALID_ARG, "theta must be finite and >= 0");
    if (!std::isfinite(c->softening) || c->softening < 0.0)
        return set_error(BH_INVALID_ARG, "softening_kpc must be finite and >= 0");
    if (!std::isfinite(c->g) || c->g <= 0.0)
        return set_error(BH_INVALID_ARG, "g must be positive and finite");
    if (c->bucket == 0 || c->bucket > 1024)
        return set_error(BH_INVALID_ARG, "bucket must be in 1..=1024");
    if (c->max_depth == 0 || c->max_depth > 128)
        return set_error(BH_INVALID_ARG, "max_depth must be in 1..=128");
    // nbody_parallel.rs:848-850: physics must stay finite as f32
    const float t = (float)c->theta, s = (float)c->softening, g = (float)c->g;
    if (!std::isfinite(t) || !std::isfinite(s) || !std::isfinite(g) || g <= 0.f)
        return set_error(BH_INVALID_ARG, "force settings are not representable as finite f32");
    return BH_OK;
}

static uint32_t eff_depth(const bh_config& c) { return std::min<uint32_t>(c.max_depth, kMortonDepth); }

// Upper bound on cells: leaves are disjoint (<= n); internal cells exist at
// depths 0..max_depth-1, and those at depth d are at most 4^d (one per
// quadtree square) and hold disjoint ranges of > bucket bodies (at most
// n/(bucket+1)).  At bucket 1 this is ~3.8n cells for n = 2^22 (a
// depth-blind n/(bucket+1) per depth would be 9n); trees of real
// distributions hold ~1.7n.
static uint64_t cell_bound(uint32_t n, const bh_config& c) {
    const uint64_t per_depth = n / ((uint64_t)c.bucket + 1);
    uint64_t internal = 0, squares = 1;
    for (uint32_t d = 0; d < eff_depth(c); ++d, squares *= 4)
        internal += std::min(squares, per_depth);
    return (uint64_t)n + internal + 1;
}

// Whether the f32 softening squared is a normal number (k_traverse's rule).
static bool normal_eps2(const bh_config* cfgs, size_t count) {
    for (size_t s = 0; s < count; ++s) {
        const float eps = (float)cfgs[s].softening;
        if (!(eps * eps >= FLT_MIN)) return false;
    }
    return true;
}

static void fill_physics(SimDesc& sd, const bh_config& c) {
    sd.bucket = c.bucket;
    sd.max_depth = eff_depth(c);
    sd.flags = c.flags;
    sd.theta = c.theta;
    sd.theta_f = (float)c.theta;
    sd.inv_theta_f = c.theta > 0.0 ? (float)(1.0 / c.theta) : INFINITY;
    sd.eps_f = (float)c.softening;
    sd.g_f = (float)c.g;
}

// ------------------------------------------------------------------- state --

struct bh_state {
    bh_device* dev = nullptr;
    uint32_t n = 0;
    GpuEvolveState* d_state = nullptr;
    float4* d_accel = nullptr;
    float* d_potential = nullptr;
    // a one-simulation layout for stand-alone kick / drift launches
    SimDesc* d_sim = nullptr;
    uint32_t* d_chunk_sim = nullptr;
    uint32_t* d_minmax = nullptr;
    double* d_cons = nullptr;  // conservation partials + result
    uint32_t* d_check = nullptr;         // first invalid record index of the last check
    GpuEvolveState* d_stage = nullptr;   // upload staging (first galaxy_bh_write_state)
    uint32_t nchunks = 0;
    SimDesc h_sim{};
};

static int enqueue_check(bh_state* st, const void* records, int kind, uint32_t n);
static int fetch_check(bh_state* st, uint32_t* first_bad);

extern "C" int galaxy_bh_state_create(bh_device* dev, const GpuEvolveState* host, uint32_t n,
                                      bh_state** out, bh_stage_timing* timing) {
    int rc = enter(dev);
    if (rc) return rc;
    if (!out || !host) return set_error(BH_INVALID_ARG, "null argument");
    *out = nullptr;
    // nbody_gpu.rs:787-789
    if (n < 2 || n > (1u << 30))
        return set_error(BH_INVALID_ARG, "GPU evolving state requires 2..=%u resident bodies",
                         1u << 30);
    bh_state* st = new bh_state();
    st->dev = dev;
    device_ref(dev);
    st->n = n;
    st->nchunks = (n + kChunk - 1) / kChunk;
    cudaEventRecord(dev->ev[0], dev->stream);
    cudaError_t e;
    std::vector<uint32_t> chunk(st->nchunks, 0u);
    auto take = [&](auto** ptr, size_t bytes) {
        return pool_alloc(dev, dev->pool, (void**)ptr, bytes);
    };
    if ((e = take(&st->d_state, sizeof(GpuEvolveState) * (size_t)n)) ||
        (e = take(&st->d_accel, sizeof(float4) * (size_t)n)) ||
        (e = take(&st->d_sim, sizeof(SimDesc))) ||
        (e = take(&st->d_chunk_sim, sizeof(uint32_t) * st->nchunks)) ||
        (e = take(&st->d_minmax, 16)) || (e = take(&st->d_check, 16))) {
        galaxy_bh_state_destroy(st);
        return cuda_fail(e, "evolving state allocation");
    }
    st->h_sim.state = st->d_state;
    st->h_sim.accel = st->d_accel;
    st->h_sim.off = 0;
    st->h_sim.n = n;
    if ((e = copy_up(dev, st->d_state, host, sizeof(GpuEvolveState) * (size_t)n)) ||
        (e = cudaMemsetAsync(st->d_accel, 0, sizeof(float4) * (size_t)n, dev->stream)) ||
        (e = cudaMemcpyAsync(st->d_chunk_sim, chunk.data(), 4 * chunk.size(),
                             cudaMemcpyHostToDevice, dev->stream)) ||
        (e = cudaMemcpyAsync(st->d_sim, &st->h_sim, sizeof(SimDesc), cudaMemcpyHostToDevice,
                             dev->stream))) {
        galaxy_bh_state_destroy(st);
        return cuda_fail(e, "evolving state upload");
    }
    cudaEventRecord(dev->ev[1], dev->stream);
    // nbody_gpu.rs:802-810: every record finite with a positive mass, tested
    // on the uploaded copy; the smallest failing index is reported and no
    // state is created
    uint32_t bad = kNone;
    if ((rc = enqueue_check(st, st->d_state, 0, n)) || (rc = fetch_check(st, &bad))) {
        galaxy_bh_state_destroy(st);
        return rc;
    }
    if (bad != kNone) {
        galaxy_bh_state_destroy(st);
        return set_error(BH_NONFINITE, "body %u contains invalid evolving state", bad);
    }
    if (timing) {
        float ms = 0.f;
        cudaEventElapsedTime(&ms, dev->ev[0], dev->ev[1]);
        *timing = bh_stage_timing{ms * 1e-3, 0.0, 0.0};
    }
    *out = st;
    return BH_OK;
}

extern "C" int galaxy_bh_state_destroy(bh_state* st) {
    if (!st) return BH_OK;
    if (st->dev) {
        cudaSetDevice(st->dev->ordinal);
        cudaStreamSynchronize(st->dev->stream);
        // back to the device's pool, in stream order (no device-wide sync)
        for (void* p : {(void*)st->d_state, (void*)st->d_accel, (void*)st->d_sim,
                        (void*)st->d_chunk_sim, (void*)st->d_minmax, (void*)st->d_check})
            if (p) cudaFreeAsync(p, st->dev->stream);
    }
    if (st->d_potential) cudaFree(st->d_potential);
    if (st->d_cons) cudaFree(st->d_cons);
    if (st->d_stage) cudaFree(st->d_stage);
    bh_device* dev = st->dev;
    delete st;
    device_unref(dev);
    return BH_OK;
}

// Hands a state made on one device handle to another handle of the same
// GPU (the serving loop's stager uploads and solves on its own handle and
// stream): the state's pending work finishes first; its buffers stay where
// they are and are later released on the new handle's stream.
int gbh::state_move(bh_state* st, bh_device* to) {
    if (!st || !to) return set_error(BH_INVALID_ARG, "null argument");
    if (st->dev == to) return BH_OK;
    if (st->dev->ordinal != to->ordinal)
        return set_error(BH_INVALID_ARG, "state and device handle are on different GPUs");
    CK(cudaSetDevice(st->dev->ordinal), "cudaSetDevice");
    CK(cudaStreamSynchronize(st->dev->stream), "state move");
    bh_device* old = st->dev;
    device_ref(to);
    st->dev = to;
    device_unref(old);
    return BH_OK;
}

extern "C" int galaxy_bh_state_count(bh_state* st, uint32_t* n) {
    if (!st || !n) return set_error(BH_INVALID_ARG, "null argument");
    *n = st->n;
    return BH_OK;
}

extern "C" int galaxy_bh_state_bytes(bh_state* st, uint64_t* bytes) {
    if (!st || !bytes) return set_error(BH_INVALID_ARG, "null argument");
    *bytes = (uint64_t)st->n * (sizeof(GpuEvolveState) + sizeof(float4));
    return BH_OK;
}

static int checked_dt(double dt, float* out) {
    if (!std::isfinite(dt) || dt <= 0.0)
        return set_error(BH_INVALID_ARG, "dt_myr must be positive and finite");
    float f = (float)dt;
    if (!std::isfinite(f) || f <= 0.f)
        return set_error(BH_INVALID_ARG, "dt_myr cannot be represented as finite f32");
    *out = f;
    return BH_OK;
}

static int stage_time(bh_device* dev, bh_stage_timing* t) {
    CK(cudaEventRecord(dev->ev[1], dev->stream), "event record");
    CK(cudaStreamSynchronize(dev->stream), "stream synchronize");
    if (t) {
        float ms = 0.f;
        cudaEventElapsedTime(&ms, dev->ev[0], dev->ev[1]);
        *t = bh_stage_timing{0.0, ms * 1e-3, 0.0};
    }
    return BH_OK;
}

static int integrate_state(bh_device* dev, bh_state* st, double dt, int mode,
                           bh_stage_timing* timing) {
    int rc = enter(dev);
    if (rc) return rc;
    if (!st || st->dev != dev) return set_error(BH_INVALID_ARG, "state does not belong to device");
    float f = 0.f;
    if ((rc = checked_dt(dt, &f))) return rc;
    st->h_sim.dt = f;
    CK(cudaMemcpyAsync(st->d_sim, &st->h_sim, sizeof(SimDesc), cudaMemcpyHostToDevice,
                       dev->stream),
       "settings upload");
    CK(cudaMemsetAsync(st->d_minmax, 0, 16, dev->stream), "memset");
    CK(cudaEventRecord(dev->ev[0], dev->stream), "event record");
    BatchBuffers b{};
    b.sims = st->d_sim;
    b.chunk_sim = st->d_chunk_sim;
    b.nchunks = st->nchunks;
    b.minmax = st->d_minmax;
    CK(launch_integrate(b, mode, dev->stream), "integrate launch");
    return stage_time(dev, timing);
}

extern "C" int galaxy_bh_kick_drift(bh_device* dev, bh_state* st, double dt,
                                    bh_stage_timing* timing) {
    return integrate_state(dev, st, dt, 1, timing);
}

extern "C" int galaxy_bh_final_kick(bh_device* dev, bh_state* st, double dt,
                                    bh_stage_timing* timing) {
    return integrate_state(dev, st, dt, 2, timing);
}

extern "C" int galaxy_bh_final_kick_drift(bh_device* dev, bh_state* st, double dt,
                                          bh_stage_timing* timing) {
    return integrate_state(dev, st, dt, 3, timing);
}

// Enqueues the record check of n records at `records` (kind 0: evolving
// states, 1: accelerations) and the copy of its result word to *first_bad.
static int enqueue_check(bh_state* st, const void* records, int kind, uint32_t n) {
    bh_device* dev = st->dev;
    CK(cudaMemsetAsync(st->d_check, 0xff, 4, dev->stream), "memset");
    CK(launch_check_records(records, kind, n, st->d_check, dev->stream), "record check");
    return BH_OK;
}

static int fetch_check(bh_state* st, uint32_t* first_bad) {
    CK(cudaMemcpyAsync(first_bad, st->d_check, 4, cudaMemcpyDeviceToHost, st->dev->stream),
       "record check readback");
    CK(cudaStreamSynchronize(st->dev->stream), "record check readback");
    return BH_OK;
}

extern "C" int galaxy_bh_read_state(bh_device* dev, bh_state* st, GpuEvolveState* out,
                                    uint32_t n, bh_stage_timing* timing) {
    int rc = enter(dev);
    if (rc) return rc;
    if (!st || !out) return set_error(BH_INVALID_ARG, "null argument");
    if (n != st->n) return set_error(BH_INVALID_ARG, "readback count %u != resident bodies %u", n, st->n);
    // nbody_gpu.rs:1043-1053 checks the host copy; the same test runs on the
    // device records (bitwise the same values) while they are copied out
    if ((rc = enqueue_check(st, st->d_state, 0, n))) return rc;
    CK(cudaEventRecord(dev->ev[0], dev->stream), "event record");
    CK(copy_down(dev, out, st->d_state, sizeof(GpuEvolveState) * (size_t)n), "state readback");
    CK(cudaEventRecord(dev->ev[1], dev->stream), "event record");
    uint32_t bad = kNone;
    if ((rc = fetch_check(st, &bad))) return rc;
    if (timing) {
        float ms = 0.f;
        cudaEventElapsedTime(&ms, dev->ev[0], dev->ev[1]);
        *timing = bh_stage_timing{0.0, 0.0, ms * 1e-3};
    }
    if (bad != kNone)
        return set_error(BH_NONFINITE, "GPU produced invalid evolving body state at %u", bad);
    return BH_OK;
}

extern "C" int galaxy_bh_read_accel(bh_device* dev, bh_state* st, GpuAccel* out, uint32_t n,
                                    bh_stage_timing* timing) {
    int rc = enter(dev);
    if (rc) return rc;
    if (!st || !out) return set_error(BH_INVALID_ARG, "null argument");
    if (n != st->n) return set_error(BH_INVALID_ARG, "readback count %u != resident bodies %u", n, st->n);
    // nbody_gpu.rs:1097-1101, evaluated on the device records
    if ((rc = enqueue_check(st, st->d_accel, 1, n))) return rc;
    CK(cudaEventRecord(dev->ev[0], dev->stream), "event record");
    CK(copy_down(dev, out, st->d_accel, sizeof(float4) * (size_t)n), "acceleration readback");
    CK(cudaEventRecord(dev->ev[1], dev->stream), "event record");
    uint32_t bad = kNone;
    if ((rc = fetch_check(st, &bad))) return rc;
    if (timing) {
        float ms = 0.f;
        cudaEventElapsedTime(&ms, dev->ev[0], dev->ev[1]);
        *timing = bh_stage_timing{0.0, 0.0, ms * 1e-3};
    }
    if (bad != kNone)
        return set_error(BH_NONFINITE, "GPU produced invalid evolving acceleration at %u", bad);
    return BH_OK;
}

extern "C" int galaxy_bh_write_state(bh_device* dev, bh_state* st, const GpuEvolveState* host,
                                     uint32_t n) {
    int rc = enter(dev);
    if (rc) return rc;
    if (!st || !host) return set_error(BH_INVALID_ARG, "null argument");
    if (n != st->n) return set_error(BH_INVALID_ARG, "write count %u != resident bodies %u", n, st->n);
    // Upload into a staging buffer, check the records there and only then
    // replace the resident state: an invalid upload leaves it untouched.
    if (!st->d_stage)
        CK(cudaMalloc(&st->d_stage, sizeof(GpuEvolveState) * (size_t)n), "staging allocation");
    CK(copy_up(dev, st->d_stage, host, sizeof(GpuEvolveState) * (size_t)n), "state upload");
    if ((rc = enqueue_check(st, st->d_stage, 0, n))) return rc;
    uint32_t bad = kNone;
    if ((rc = fetch_check(st, &bad))) return rc;
    if (bad != kNone) return set_error(BH_NONFINITE, "body %u contains invalid evolving state", bad);
    CK(cudaMemcpyAsync(st->d_state, st->d_stage, sizeof(GpuEvolveState) * (size_t)n,
                       cudaMemcpyDeviceToDevice, dev->stream),
       "state upload");
    return BH_OK;
}

static int ensure_potential(bh_state* st) {
    if (!st->d_potential) {
        CK(cudaMalloc(&st->d_potential, sizeof(float) * (size_t)st->n), "potential allocation");
        CK(cudaMemsetAsync(st->d_potential, 0, sizeof(float) * (size_t)st->n, st->dev->stream),
           "memset");
    }
    return BH_OK;
}

extern "C" int galaxy_bh_direct_probes(bh_device* dev, bh_state* st, const bh_config* cfg,
                                       const uint32_t* probes, uint32_t nprobes, double* out) {
    int rc = enter(dev);
    if (rc) return rc;
    if (!st || !cfg || !probes || !out) return set_error(BH_INVALID_ARG, "null argument");
    if ((rc = validate_config(cfg))) return rc;
    if (nprobes == 0) return BH_OK;
    for (uint32_t k = 0; k < nprobes; ++k)
        if (probes[k] >= st->n) return set_error(BH_INVALID_ARG, "body index is out of range");
    const size_t sums = 16ull * nprobes * probe_slices(st->n, nprobes);
    PoolBlock block(dev);
    cudaError_t e = block.get(sums + 4ull * nprobes);
    double* d_o = reinterpret_cast<double*>(block.at);
    uint32_t* d_p = reinterpret_cast<uint32_t*>(block.at + sums);
    if (!e) e = cudaMemcpyAsync(d_p, probes, 4ull * nprobes, cudaMemcpyHostToDevice, dev->stream);
    if (!e)
        e = launch_direct_probes(st->d_state, st->n, d_p, nprobes, cfg->softening, cfg->g, d_o,
                                 dev->stream);
    if (!e) e = copy_down(dev, out, d_o, 16ull * nprobes);
    if (!e) e = block.wait();
    if (e) return cuda_fail(e, "direct probes");
    return BH_OK;
}

extern "C" int galaxy_bh_conservation(bh_device* dev, bh_state* st, double out[10]) {
    int rc = enter(dev);
    if (rc) return rc;
    if (!st || !out) return set_error(BH_INVALID_ARG, "null argument");
    const uint32_t nb = conservation_blocks(st->n);
    if (!st->d_cons) CK(cudaMalloc(&st->d_cons, sizeof(double) * (9 * (size_t)nb + 16)), "alloc");
    CK(launch_conservation(st->d_state, st->d_potential, st->n, st->d_cons, nb,
                           st->d_cons + 9 * (size_t)nb, dev->stream),
       "conservation launch");
    double r[9];
    CK(cudaMemcpyAsync(r, st->d_cons + 9 * (size_t)nb, sizeof r, cudaMemcpyDeviceToHost,
                       dev->stream),
       "readback");
    CK(cudaStreamSynchronize(dev->stream), "conservation");
    out[0] = r[0];
    out[1] = r[1] / r[0];
    out[2] = r[2] / r[0];
    out[3] = r[3];
    out[4] = r[4];
    out[5] = r[5];
    out[6] = r[6];
    out[7] = r[7];
    out[8] = r[8];
    out[9] = r[6] + r[7];
    return BH_OK;
}

// ------------------------------------------------------------------- batch --

struct Batch {
    bh_device* dev = nullptr;
    std::vector<bh_state*> states;
    std::vector<bh_config> cfgs;
    std::vector<SimDesc> h_sims;
    std::vector<uint32_t> h_chunk_sim;
    std::vector<Tile> h_tiles;
    uint32_t npos = 0, nchunks = 0, ntiles = 0, nscan_tiles = 0;
    uint64_t cell_capacity = 0;
    void* arena = nullptr;
    size_t arena_bytes = 0;
    void* control = nullptr;
    size_t control_bytes = 0;
    BatchBuffers bb{};
    SimDesc* d_sims = nullptr;
    // graphs: [0] first step, [1] middle step, [2] final kick
    cudaGraphExec_t graphs[3] = {nullptr, nullptr, nullptr};
    uint32_t graph_flags = 0xffffffffu;
    bool stats_valid = false;
    // theta and G the cell records (G*m, MAC bounds) were last computed with
    // (single-simulation trees; batches keep their creation configs)
    double built_theta = NAN, built_g = NAN;

    size_t arena_capacity = 0;  // bytes held

    ~Batch() {
        for (auto& g : graphs)
            if (g) cudaGraphExecDestroy(g);
        // back to the device handle's pool in stream order: no device-wide
        // synchronisation (a cudaFree would wait for every stream of the GPU,
        // e.g. a serving loop's rounds while its stager releases a tree)
        if (arena) cudaFreeAsync(arena, dev->stream);
    }
};

struct Layout {
    uint32_t npos = 0, nchunks = 0, ntiles = 0, nscan_tiles = 0;
    uint64_t cells = 0;
    std::vector<uint32_t> off;
};

static Layout plan_layout(const uint32_t* counts, const bh_config* cfgs, uint32_t count) {
    Layout L;
    uint64_t pos = 0;
    L.off.resize(count);
    for (uint32_t s = 0; s < count; ++s) {
        L.off[s] = (uint32_t)pos;
        pos += (counts[s] + kChunk - 1) / kChunk * kChunk;
        L.ntiles += (counts[s] + kTile - 1) / kTile;
        L.cells += cell_bound(counts[s], cfgs[s]);
    }
    L.npos = (uint32_t)pos;
    L.nchunks = L.npos / kChunk;
    L.nscan_tiles = (L.npos + 1 + kScanTile - 1) / kScanTile;
    return L;
}

static size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

// Byte sizes of the arena regions, in carve order.
struct ArenaPlan {
    size_t control, sims, simout, chunk, tiles, keys, vals, sbody, base, cell_u, groups,
        cell_d, agg_region, err, stats;
    size_t total() const {
        return control + sims + simout + chunk + tiles + 2 * keys + 2 * vals + sbody + base +
               cell_u + groups + cell_d + agg_region + err + stats;
    }
};

static ArenaPlan plan_arena(const Layout& L, uint32_t nsims) {
    ArenaPlan a;
    a.control = align256(4ull * nsims * 4 + 4ull * nsims * kRadixPasses * kRadixDigits + 4ull * 32 +
                         4ull * kRadixPasses * L.ntiles * kRadixDigits) +
                align256(8ull * L.nscan_tiles);
    a.sims = align256(sizeof(SimDesc) * nsims);
    a.simout = align256(sizeof(SimOut) * nsims);
    a.chunk = align256(4ull * L.nchunks);
    a.tiles = align256(sizeof(Tile) * L.ntiles);
    a.keys = align256(4ull * L.npos);
    a.vals = align256(4ull * L.npos);
    a.sbody = align256(16ull * L.npos);
    a.base = align256(4ull * (L.npos + 1));
    a.cell_u = align256(sizeof(uint4) * L.cells);
    a.groups = align256(4ull * sizeof(CellRec) * (L.cells + nsims));
    a.cell_d = align256(32ull * L.cells);
    // far more than the lists need: the arena's size is part of the receipts
    a.agg_region = align256(16ull * L.cells) + 2 * align256(4ull * L.cells);
    a.err = 256;
    a.stats = 256;
    return a;
}

extern "C" int galaxy_bh_batch_footprint(const uint32_t* counts, const bh_config* cfgs,
                                         uint32_t count, uint64_t* bytes) {
    if (!counts || !cfgs || !bytes || !count) return set_error(BH_INVALID_ARG, "null argument");
    Layout L = plan_layout(counts, cfgs, count);
    uint64_t persistent = 0;
    for (uint32_t s = 0; s < count; ++s)
        persistent += (uint64_t)counts[s] * (sizeof(GpuEvolveState) + sizeof(float4) + 4) +
                      ((counts[s] + 31) / 32) * 4 + 1024;
    *bytes = plan_arena(L, count).total() + persistent;
    return BH_OK;
}

// Builds a batch of `count` states.  A `donor` batch of the same device
// handle (or null) gives up its arena when that is large enough, and is
// freed either way: re-forming a batch, or pointing a tree at another state,
// then allocates nothing (the donor's work precedes the new batch's on the
// handle's stream).
static int batch_build(bh_device* dev, bh_state* const* states, const bh_config* cfgs,
                       uint32_t count, Batch** out, Batch* donor_batch = nullptr) {
    std::unique_ptr<Batch> donor(donor_batch);
    *out = nullptr;
    if (!count) return set_error(BH_INVALID_ARG, "batch needs at least one state");
    std::vector<uint32_t> counts(count);
    for (uint32_t s = 0; s < count; ++s) {
        if (!states[s] || states[s]->dev != dev)
            return set_error(BH_INVALID_ARG, "state %u does not belong to this device", s);
        int rc = validate_config(&cfgs[s]);
        if (rc) return rc;
        counts[s] = states[s]->n;
    }
    Layout L = plan_layout(counts.data(), cfgs, count);
    if (L.cells >= (1ull << 31) || (uint64_t)L.npos + 1 >= (1ull << 31))
        return set_error(BH_CAPACITY_OVERFLOW, "batch exceeds 2^31 positions or cells");
    ArenaPlan A = plan_arena(L, count);
    Batch* b = new Batch();
    b->dev = dev;
    b->states.assign(states, states + count);
    b->cfgs.assign(cfgs, cfgs + count);
    b->npos = L.npos;
    b->nchunks = L.nchunks;
    b->ntiles = L.ntiles;
    b->nscan_tiles = L.nscan_tiles;
    b->cell_capacity = L.cells;
    b->arena_bytes = A.total();
    cudaError_t e = cudaSuccess;
    if (donor && donor->arena && donor->arena_capacity >= b->arena_bytes) {
        b->arena = donor->arena;
        b->arena_capacity = donor->arena_capacity;
        donor->arena = nullptr;
    }
    donor.reset();  // a donor arena too small goes back to the pool first
    // the arena comes from the device handle's stream-ordered pool, which
    // keeps released arenas and state buffers for reuse
    if (!b->arena) {
        e = pool_alloc(dev, dev->pool, &b->arena, b->arena_bytes);
        b->arena_capacity = b->arena_bytes;
    }
    if (e != cudaSuccess) {
        delete b;
        return cuda_fail(e, "batch arena allocation");
    }
    char* p = (char*)b->arena;
    auto take = [&](size_t bytes) {
        char* q = p;
        p += bytes;
        return (void*)q;
    };
    BatchBuffers& bb = b->bb;
    b->control = p;
    b->control_bytes = A.control;
    char* cp = (char*)take(A.control);
    bb.minmax = (uint32_t*)cp;
    cp += 4ull * count * 4;
    bb.hist = (uint32_t*)cp;
    cp += 4ull * count * kRadixPasses * kRadixDigits;
    bb.counters = (uint32_t*)cp;
    cp += 4ull * 32;
    bb.sort_flags = (uint32_t*)cp;
    cp += 4ull * kRadixPasses * L.ntiles * kRadixDigits;
    bb.scan_flags = (unsigned long long*)((char*)b->control +
                                          align256((size_t)(cp - (char*)b->control)));
    b->d_sims = (SimDesc*)take(A.sims);
    bb.sims = b->d_sims;
    bb.simout = (SimOut*)take(A.simout);
    bb.chunk_sim = (const uint32_t*)take(A.chunk);
    bb.tiles = (const Tile*)take(A.tiles);
    bb.keys_a = (uint32_t*)take(A.keys);
    bb.keys_b = (uint32_t*)take(A.keys);
    bb.vals_a = (uint32_t*)take(A.vals);
    bb.vals_b = (uint32_t*)take(A.vals);
    bb.sbody = (float4*)take(A.sbody);
    bb.base = (uint32_t*)take(A.base);
    bb.cell_u = (uint4*)take(A.cell_u);
    bb.groups = (CellRec*)take(A.groups);
    bb.cell_d = (double4*)take(A.cell_d);
    bb.agg_region = take(A.agg_region);
    bb.err = (uint32_t*)take(A.err);
    bb.force_stats = (unsigned long long*)take(A.stats);
    bb.nsims = count;
    bb.max_bodies = *std::max_element(counts.begin(), counts.end());
    bb.npos = L.npos;
    bb.nchunks = L.nchunks;
    bb.ntiles = L.ntiles;
    bb.nscan_tiles = L.nscan_tiles;
    bb.cell_capacity = (uint32_t)L.cells;
    bb.radix_bits = 8;
    bb.trav_warps = 4;
    bb.clusters = true;
    bb.normal_eps2 = normal_eps2(cfgs, count);

    b->h_sims.resize(count);
    b->h_chunk_sim.assign(L.nchunks, kNone);
    uint32_t tile = 0, group = 0;
    for (uint32_t s = 0; s < count; ++s) {
        SimDesc& sd = b->h_sims[s];
        memset(&sd, 0, sizeof sd);
        sd.state = states[s]->d_state;
        sd.accel = states[s]->d_accel;
        sd.potential = states[s]->d_potential;
        sd.off = L.off[s];
        sd.n = counts[s];
        sd.first_tile = tile;
        sd.dt = 0.f;
        fill_physics(sd, cfgs[s]);
        for (uint32_t c = 0; c < (counts[s] + kChunk - 1) / kChunk; ++c)
            b->h_chunk_sim[L.off[s] / kChunk + c] = s;
        for (uint32_t t0 = 0; t0 < counts[s]; t0 += kTile) {
            Tile tl{};
            tl.sim = s;
            tl.start = L.off[s] + t0;
            tl.count = std::min<uint32_t>(kTile, counts[s] - t0);
            // 8 KB per group of simulations above kTile bodies: agg_region has 96
            tl.group = counts[s] <= kTile ? kNone : group + t0 / (kTile * kGroupTiles);
            b->h_tiles.push_back(tl);
            ++tile;
        }
        if (counts[s] > kTile) group += (counts[s] + kTile * kGroupTiles - 1) / (kTile * kGroupTiles);
    }
    cudaStream_t st = dev->stream;
    if ((e = cudaMemcpyAsync(b->d_sims, b->h_sims.data(), sizeof(SimDesc) * count,
                             cudaMemcpyHostToDevice, st)) ||
        (e = cudaMemcpyAsync((void*)bb.chunk_sim, b->h_chunk_sim.data(), 4ull * L.nchunks,
                             cudaMemcpyHostToDevice, st)) ||
        (e = cudaMemcpyAsync((void*)bb.tiles, b->h_tiles.data(), sizeof(Tile) * L.ntiles,
                             cudaMemcpyHostToDevice, st)) ||
        (e = cudaMemsetAsync(bb.err, 0, 256, st)) ||
        (e = cudaMemsetAsync(bb.force_stats, 0, 256, st)) ||
        (e = cudaMemsetAsync(bb.simout, 0, sizeof(SimOut) * count, st)) ||
        (e = cudaStreamSynchronize(st))) {
        delete b;
        return cuda_fail(e, "batch upload");
    }
    *out = b;
    return BH_OK;
}

static int upload_sims(Batch* b) {
    CK(cudaMemcpyAsync(b->d_sims, b->h_sims.data(), sizeof(SimDesc) * b->h_sims.size(),
                       cudaMemcpyHostToDevice, b->dev->stream),
       "settings upload");
    return BH_OK;
}

// Reads (and clears) the device error word; maps bits to a status.  stage_cycles
// (or null): kStages words, as the last timed small sort left them.
static int check_device_errors(Batch* b, uint32_t* stage_cycles = nullptr) {
    uint32_t words[kStageCycles + kStages] = {};
    CK(cudaMemcpyAsync(words, b->bb.err, stage_cycles ? sizeof words : 4, cudaMemcpyDeviceToHost,
                       b->dev->stream),
       "readback");
    CK(cudaStreamSynchronize(b->dev->stream), "stream synchronize");
    const uint32_t err = words[0];
    if (stage_cycles) std::copy_n(words + kStageCycles, kStages, stage_cycles);
    if (!err) return BH_OK;
    cudaMemsetAsync(b->bb.err, 0, 4, b->dev->stream);
    cudaStreamSynchronize(b->dev->stream);
    if (err & kErrLookbackTimeout)
        return set_error(BH_TIMEOUT, "device look-back wait timed out (error bits 0x%x)", err);
    if (err & kErrCapacity)
        return set_error(BH_CAPACITY_OVERFLOW, "GPU tree reported cell-capacity overflow");
    return set_error(BH_CUDA_ERROR, "device traversal reported error bits 0x%x", err);
}

enum Stage { kStBounds, kStMorton, kStRadix, kStTopology, kStAggregate };

// memset(control) + bounds/integrate + Morton + radix + topology + aggregates.
// With ev != null, records events between stages (ev[0..5]).
static int enqueue_rebuild(Batch* b, int integrate_mode, cudaEvent_t* ev) {
    cudaStream_t s = b->dev->stream;
    if (ev) CK(cudaEventRecord(ev[0], s), "event");
    const bool small = small_sort(b->bb);  // one launch
    const bool scanned = small && b->bb.nsims == 1;
    if (!scanned) CK(cudaMemsetAsync(b->control, 0, b->control_bytes, s), "control memset");
    if (!small) CK(launch_integrate(b->bb, integrate_mode, s), "integrate launch");
    if (ev) CK(cudaEventRecord(ev[1], s), "event");
    if (!small) CK(launch_morton(b->bb, s), "morton launch");
    if (ev) CK(cudaEventRecord(ev[2], s), "event");
    CK(small ? launch_sort_small(b->bb, integrate_mode, ev != nullptr, s) : launch_radix(b->bb, s), "radix launch");
    if (ev) CK(cudaEventRecord(ev[3], s), "event");
    if (!scanned) CK(launch_count_scan(b->bb, s), "count/scan launch");
    if (ev) CK(cudaEventRecord(ev[4], s), "event");
    CK(launch_aggregate(b->bb, s), "aggregate launch");
    if (ev) CK(cudaEventRecord(ev[5], s), "event");
    return BH_OK;
}

static bool any_flag(Batch* b, uint32_t flag) {
    for (auto& c : b->cfgs)
        if (c.flags & flag) return true;
    return false;
}

static bool any_without_flag(Batch* b, uint32_t flag) {
    for (auto& c : b->cfgs)
        if (!(c.flags & flag)) return true;
    return false;
}

static int enqueue_force(Batch* b, bool stats) {
    cudaStream_t s = b->dev->stream;
    if (stats) CK(cudaMemsetAsync(b->bb.force_stats, 0, 40, s), "memset");
    CK(launch_traverse(b->bb, any_flag(b, BH_FLAG_COMPENSATED),
                       any_without_flag(b, BH_FLAG_COMPENSATED), any_flag(b, BH_FLAG_POTENTIAL),
                       stats, s),
       "traverse launch");
    return BH_OK;
}

// Installs per-simulation configs.  A rebuild under a config needing more
// cells than the arena holds must be preceded by tree_fit.
static int apply_configs(Batch* b, const bh_config* cfgs, bool for_rebuild) {
    for (size_t s = 0; s < b->states.size(); ++s) {
        int rc = validate_config(&cfgs[s]);
        if (rc) return rc;
        if (for_rebuild && cell_bound(b->states[s]->n, cfgs[s]) > b->cell_capacity)
            return set_error(BH_CAPACITY_OVERFLOW,
                             "config needs more tree cells than this tree holds");
        if (cfgs[s].flags & BH_FLAG_POTENTIAL) {
            if ((rc = ensure_potential(b->states[s]))) return rc;
        }
        b->cfgs[s] = cfgs[s];
        b->h_sims[s].potential = b->states[s]->d_potential;
        fill_physics(b->h_sims[s], cfgs[s]);
    }
    b->bb.normal_eps2 = normal_eps2(b->cfgs.data(), b->cfgs.size());
    return upload_sims(b);
}

static int run_graphs(Batch* b, uint32_t nsteps) {
    cudaStream_t s = b->dev->stream;
    const uint32_t flags = (any_flag(b, BH_FLAG_COMPENSATED) ? 1u : 0u) |
                           (any_flag(b, BH_FLAG_POTENTIAL) ? 2u : 0u) |
                           (any_without_flag(b, BH_FLAG_COMPENSATED) ? 4u : 0u) |
                           (b->bb.normal_eps2 ? 8u : 0u);
    if (b->graph_flags != flags) {
        for (auto& g : b->graphs)
            if (g) {
                cudaGraphExecDestroy(g);
                g = nullptr;
            }
        for (int k = 0; k < 3; ++k) {
            cudaGraph_t graph;
            CK(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal), "begin capture");
            int rc = BH_OK;
            if (k < 2) {
                rc = enqueue_rebuild(b, k == 0 ? 1 : 3, nullptr);
                if (!rc) rc = enqueue_force(b, false);
            } else {
                cudaError_t e = launch_integrate(b->bb, 2, s);
                if (e) rc = cuda_fail(e, "integrate launch");
            }
            cudaError_t e = cudaStreamEndCapture(s, &graph);
            if (rc) return rc;
            CK(e, "end capture");
            e = cudaGraphInstantiate(&b->graphs[k], graph, 0);
            cudaGraphDestroy(graph);
            CK(e, "graph instantiate");
        }
        b->graph_flags = flags;
    }
    for (uint32_t k = 0; k < nsteps; ++k)
        CK(cudaGraphLaunch(b->graphs[k == 0 ? 0 : 1], s), "graph launch");
    CK(cudaGraphLaunch(b->graphs[2], s), "graph launch");
    b->stats_valid = false;
    return check_device_errors(b);
}

// -------------------------------------------------------------------- tree --

struct bh_tree {
    bh_device* dev = nullptr;
    bh_state* st = nullptr;
    Batch* batch = nullptr;
    bool built = false;
};

extern "C" int galaxy_bh_tree_create(bh_device* dev, bh_state* st, const bh_config* cfg,
                                     bh_tree** out) {
    int rc = enter(dev);
    if (rc) return rc;
    if (!out || !st) return set_error(BH_INVALID_ARG, "null argument");
    *out = nullptr;
    if ((rc = validate_config(cfg))) return rc;
    if (st->dev != dev) return set_error(BH_INVALID_ARG, "state does not belong to device");
    Batch* b = nullptr;
    if ((rc = batch_build(dev, &st, cfg, 1, &b))) return rc;
    bh_tree* t = new bh_tree();
    t->dev = dev;
    device_ref(dev);
    t->st = st;
    t->batch = b;
    *out = t;
    return BH_OK;
}

extern "C" int galaxy_bh_tree_destroy(bh_tree* tree) {
    if (!tree) return BH_OK;
    cudaSetDevice(tree->dev->ordinal);
    cudaStreamSynchronize(tree->dev->stream);
    delete tree->batch;
    bh_device* dev = tree->dev;
    delete tree;
    device_unref(dev);
    return BH_OK;
}

// Points *tree at state st under cfg (creating the tree when null), keeping
// its arena when that is large enough: a serving loop's stager solves each
// newcomer's boundary on one tree instead of allocating one per request.  Its
// rebuilds share the GPU with the loop's rounds, so they use no cluster.
int gbh::tree_retarget(bh_device* dev, bh_tree** tree, bh_state* st, const bh_config* cfg) {
    if (!tree) return set_error(BH_INVALID_ARG, "null argument");
    int rc;
    if (!*tree) {
        if ((rc = galaxy_bh_tree_create(dev, st, cfg, tree)) == BH_OK)
            (*tree)->batch->bb.clusters = false;
        return rc;
    }
    if ((rc = enter(dev))) return rc;
    bh_tree* t = *tree;
    if (!st) return set_error(BH_INVALID_ARG, "null argument");
    if (t->dev != dev || st->dev != dev)
        return set_error(BH_INVALID_ARG, "tree or state belongs to another device handle");
    if ((rc = validate_config(cfg))) return rc;
    Batch* b = nullptr;
    Batch* donor = t->batch;
    t->batch = nullptr;
    t->built = false;
    if ((rc = batch_build(dev, &st, cfg, 1, &b, donor))) {
        galaxy_bh_tree_destroy(t);
        *tree = nullptr;
        return rc;
    }
    b->bb.clusters = false;
    t->batch = b;
    t->st = st;
    return BH_OK;
}

static int tree_check(bh_device* dev, bh_state* st, bh_tree* tree) {
    int rc = enter(dev);
    if (rc) return rc;
    if (!tree || !st) return set_error(BH_INVALID_ARG, "null argument");
    if (tree->st != st || tree->dev != dev)
        return set_error(BH_INVALID_ARG, "tree count does not match evolving state");
    return BH_OK;
}

// Re-carves the tree's arena when cfg needs more cells than it holds.
static int tree_fit(bh_tree* tree, const bh_config* cfg) {
    int rc = validate_config(cfg);
    if (rc) return rc;
    if (cell_bound(tree->st->n, *cfg) <= tree->batch->cell_capacity) return BH_OK;
    Batch* nb = nullptr;
    if ((rc = batch_build(tree->dev, &tree->st, cfg, 1, &nb))) return rc;
    nb->bb.radix_bits = tree->batch->bb.radix_bits;  // keep the tree's tuning
    nb->bb.trav_warps = tree->batch->bb.trav_warps;
    nb->bb.clusters = tree->batch->bb.clusters;
    delete tree->batch;
    tree->batch = nb;
    tree->built = false;
    return BH_OK;
}

extern "C" int galaxy_bh_tree_rebuild(bh_device* dev, bh_state* st, bh_tree* tree,
                                      const bh_config* cfg, bh_build_timing* timing) {
    int rc = tree_check(dev, st, tree);
    if (rc) return rc;
    if ((rc = tree_fit(tree, cfg))) return rc;
    if ((rc = apply_configs(tree->batch, cfg, true))) return rc;
    tree->built = false;  // until this rebuild has ended without an error
    if ((rc = enqueue_rebuild(tree->batch, 0, timing ? dev->ev : nullptr))) return rc;
    CK(cudaStreamSynchronize(dev->stream), "rebuild");
    uint32_t cycles[kStages];
    if ((rc = check_device_errors(tree->batch, cycles))) return rc;
    if (timing) {
        float ms[5];
        for (int k = 0; k < 5; ++k) cudaEventElapsedTime(&ms[k], dev->ev[k], dev->ev[k + 1]);
        if (small_sort(tree->batch->bb)) {  // one launch: divided as its own cycles are
            const float launch = ms[0] + ms[1] + ms[2] + ms[3];
            double all = 0.0;
            for (uint32_t c : cycles) all += c;
            for (uint32_t k = 0; k < kStages; ++k)
                ms[k] = all > 0.0 ? (float)(launch * (cycles[k] / all)) : 0.f;
        }
        timing->bounds_seconds = ms[0] * 1e-3;
        timing->morton_seconds = ms[1] * 1e-3;
        timing->radix_seconds = ms[2] * 1e-3;
        timing->positions_seconds = 0.0;  // fused into the last radix pass
        timing->topology_seconds = ms[3] * 1e-3;
        timing->aggregate_seconds = ms[4] * 1e-3;
    }
    tree->built = true;
    tree->batch->built_theta = cfg->theta;
    tree->batch->built_g = cfg->g;
    return BH_OK;
}

extern "C" int galaxy_bh_force(bh_device* dev, bh_state* st, bh_tree* tree, const bh_config* cfg,
                               bh_stage_timing* timing) {
    int rc = tree_check(dev, st, tree);
    if (rc) return rc;
    if (!tree->built) return set_error(BH_INVALID_ARG, "force requires a rebuilt tree");
    if ((rc = apply_configs(tree->batch, cfg, false))) return rc;
    Batch* b = tree->batch;
    if (cfg->theta != b->built_theta || cfg->g != b->built_g) {
        CK(launch_refresh_mac(b->bb, 0, dev->stream), "refresh launch");
        b->built_theta = cfg->theta;
        b->built_g = cfg->g;
    }
    CK(cudaEventRecord(dev->ev[0], dev->stream), "event");
    const bool stats = !(cfg->flags & BH_FLAG_NO_STATS);
    if ((rc = enqueue_force(tree->batch, stats))) return rc;
    if ((rc = stage_time(dev, timing))) return rc;
    tree->batch->stats_valid = stats;
    return check_device_errors(tree->batch);
}

extern "C" int galaxy_bh_force_stats(bh_device* dev, bh_tree* tree, bh_force_stats* out) {
    int rc = enter(dev);
    if (rc) return rc;
    if (!tree || !out) return set_error(BH_INVALID_ARG, "null argument");
    if (!tree->batch->stats_valid)
        return set_error(BH_INVALID_ARG, "no force statistics since the last galaxy_bh_force");
    unsigned long long v[5];
    CK(cudaMemcpyAsync(v, tree->batch->bb.force_stats, sizeof v, cudaMemcpyDeviceToHost,
                       dev->stream),
       "readback");
    CK(cudaStreamSynchronize(dev->stream), "readback");
    out->visited_nodes = v[0];
    out->approximated_cells = v[1];
    out->direct_terms = v[2];
    out->exact_mac_fallbacks = v[3];
    out->warp_iterations = v[4];
    return BH_OK;
}

extern "C" int galaxy_bh_force_f64(bh_device* dev, bh_state* st, bh_tree* tree,
                                   const bh_config* cfg, double* accel, double* abs_sum,
                                   bh_force_stats* stats) {
    int rc = tree_check(dev, st, tree);
    if (rc) return rc;
    if (!cfg || !accel) return set_error(BH_INVALID_ARG, "null argument");
    if ((rc = validate_config(cfg))) return rc;
    if (!tree->built) return set_error(BH_INVALID_ARG, "force requires a rebuilt tree");
    const size_t n = st->n;
    const size_t bytes = 16 * n + (abs_sum ? 8 * n : 0) + 32;
    PoolBlock block(dev);
    CK(block.get(bytes), "f64 traversal allocation");
    char* d = block.at;
    double* d_acc = reinterpret_cast<double*>(d);
    double* d_abs = abs_sum ? reinterpret_cast<double*>(d + 16 * n) : nullptr;
    unsigned long long* d_stats = reinterpret_cast<unsigned long long*>(d + bytes - 32);
    unsigned long long h_stats[3] = {0, 0, 0};
    cudaError_t e = cudaMemsetAsync(d_stats, 0, 32, dev->stream);
    if (!e)
        e = launch_traverse_f64(tree->batch->bb, 0, st->n, cfg->theta, cfg->softening, cfg->g,
                                d_acc, d_abs, d_stats, dev->stream);
    if (!e) e = copy_down(dev, accel, d_acc, 16 * n);
    if (!e && abs_sum) e = copy_down(dev, abs_sum, d_abs, 8 * n);
    if (!e) e = cudaMemcpyAsync(h_stats, d_stats, 24, cudaMemcpyDeviceToHost, dev->stream);
    if (!e) e = block.wait();
    if (e) return cuda_fail(e, "f64 traversal");
    if (stats) {
        *stats = bh_force_stats{};
        stats->visited_nodes = h_stats[0];
        stats->approximated_cells = h_stats[1];
        stats->direct_terms = h_stats[2];
    }
    return BH_OK;
}

// The rest of a step behind a wait that gave up, on a small simulation: its tree
// is sound when the error word is set, so what runs reads nothing out of place, but
// a rebuild has to leave the cells alone and a force to find nothing to sum.
static int probe_stalled_step(bh_device* dev) {
    constexpr uint32_t kBodies = 70000;  // sorted by tiles, with cells across outer cuts
    std::vector<GpuEvolveState> records(kBodies);
    for (uint32_t i = 0; i < kBodies; ++i) {
        records[i] = GpuEvolveState{};
        records[i].position_mass[0] = (float)(i * 2654435761u >> 8);
        records[i].position_mass[1] = (float)(i * 40503u % 65536u);
        records[i].position_mass[2] = 1.f;
    }
    const bh_config cfg{0.5, 1.0, 1.0, 4, 16, BH_FLAG_NO_STATS, 0};
    bh_state* st = nullptr;
    bh_tree* tree = nullptr;
    int rc = galaxy_bh_state_create(dev, records.data(), kBodies, &st, nullptr);
    if (!rc) rc = galaxy_bh_tree_create(dev, st, &cfg, &tree);
    if (!rc) rc = galaxy_bh_tree_rebuild(dev, st, tree, &cfg, nullptr);
    if (!rc) rc = galaxy_bh_force(dev, st, tree, &cfg, nullptr);
    std::vector<uint32_t> accel(4 * (size_t)kBodies), cells(4 * (size_t)kBodies);
    if (!rc) {
        Batch* b = tree->batch;
        cudaStream_t s = dev->stream;
        const size_t bytes = 16ull * kBodies;
        const uint32_t bits = kErrLookbackTimeout;
        cudaError_t e;
        if ((e = cudaMemsetAsync(b->bb.cell_u, 0x5a, bytes, s)) ||
            (e = cudaMemcpyAsync(b->bb.err, &bits, 4, cudaMemcpyHostToDevice, s)))
            rc = cuda_fail(e, "wait probe");
        if (!rc) rc = enqueue_rebuild(b, 0, nullptr);
        if (!rc) rc = enqueue_force(b, false);
        if (!rc && ((e = cudaMemcpyAsync(accel.data(), st->d_accel, bytes, cudaMemcpyDeviceToHost, s)) ||
                    (e = cudaMemcpyAsync(cells.data(), b->bb.cell_u, bytes, cudaMemcpyDeviceToHost, s))))
            rc = cuda_fail(e, "wait probe");
        if (!rc) rc = check_device_errors(b);
        for (size_t k = 0; rc == BH_TIMEOUT && k < cells.size(); ++k)
            if (cells[k] != 0x5a5a5a5au || accel[k] != 0u)
                rc = set_error(BH_CUDA_ERROR, "wait probe: a step went on behind a wait that gave up");
    }
    if (tree) galaxy_bh_tree_destroy(tree);
    if (st) galaxy_bh_state_destroy(st);
    return rc;
}

extern "C" int galaxy_bh_wait_probe(bh_device* dev, uint64_t spin_cycles) {
    int rc = enter(dev);
    if (rc) return rc;
    if (spin_cycles > (uint64_t)4000000000ull)
        return set_error(BH_INVALID_ARG, "spin_cycles above 4e9 (about two seconds)");
    // the words of the tile and of the groups before, two error words, the results
    constexpr size_t kBefore = kRadixDigits + 2 * kGroupStride, kResults = 2 * kRadixDigits;
    PoolBlock block(dev);
    CK(block.get((kBefore + 2 + kResults) * 4), "probe allocation");
    uint32_t* d = reinterpret_cast<uint32_t*>(block.at);
    cudaError_t e = cudaMemsetAsync(d, 0, (kBefore + 2 + kResults) * 4, dev->stream);
    if (e == cudaSuccess)
        e = launch_wait_probe(d, d + kBefore, (long long)spin_cycles, d + kBefore + 2, dev->stream);
    uint32_t got[2 + kResults] = {};
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(got, d + kBefore, sizeof got, cudaMemcpyDeviceToHost, dev->stream);
    if (e == cudaSuccess) e = block.wait();
    if (e != cudaSuccess) return cuda_fail(e, "wait probe");
    const uint32_t err = got[0] & got[1];
    bool sums = true;  // each wait returns what had been published: nothing, and 1 a digit
    for (size_t k = 0; k < kResults; ++k) sums = sums && got[2 + k] == k / kRadixDigits;
    if (!(err & kErrLookbackTimeout) || !sums)
        return set_error(BH_CUDA_ERROR, "wait probe: a bounded wait did not report its timeout");
    if ((rc = probe_stalled_step(dev)) != BH_TIMEOUT)
        return rc ? rc : set_error(BH_CUDA_ERROR, "wait probe: a stalled step reported no timeout");
    return set_error(BH_TIMEOUT,
                     "device waits (look-back over tiles, over tile groups) timed out (error bits "
                     "0x%x)",
                     err);
}

extern "C" int galaxy_bh_read_tree_evidence(bh_device* dev, bh_tree* tree, TreeMeta* meta,
                                            GpuEntry* entries, GpuBody* bodies, uint32_t n,
                                            GpuCell* cells, uint32_t cell_capacity,
                                            uint32_t* cell_count) {
    int rc = enter(dev);
    if (rc) return rc;
    if (!tree) return set_error(BH_INVALID_ARG, "null tree");
    if (!tree->built) return set_error(BH_INVALID_ARG, "tree has not been rebuilt");
    Batch* b = tree->batch;
    const uint32_t sn = tree->st->n;
    if ((entries || bodies) && n != sn)
        return set_error(BH_INVALID_ARG, "evidence count %u != resident bodies %u", n, sn);
    cudaStream_t s = dev->stream;
    uint32_t cb_ce[2];
    CK(cudaMemcpyAsync(&cb_ce[0], b->bb.base + b->h_sims[0].off, 4, cudaMemcpyDeviceToHost, s), "readback");
    CK(cudaMemcpyAsync(&cb_ce[1], b->bb.base + b->h_sims[0].off + sn, 4, cudaMemcpyDeviceToHost, s), "readback");
    SimOut so;
    CK(cudaMemcpyAsync(&so, b->bb.simout, sizeof so, cudaMemcpyDeviceToHost, s), "readback");
    CK(cudaStreamSynchronize(s), "readback");
    const uint32_t ncell = cb_ce[1] - cb_ce[0];
    if (cell_count) *cell_count = ncell;
    if (meta) {
        meta->data[0] = ncell;
        meta->data[1] = sn;
        meta->data[2] = b->h_sims[0].max_depth;
        meta->data[3] = 0;
        meta->bounds[0] = (float)so.cx;
        meta->bounds[1] = (float)so.cy;
        meta->bounds[2] = (float)so.half;
        meta->bounds[3] = 0.f;
    }
    if (cells && cell_capacity < ncell)
        return set_error(BH_CAPACITY_OVERFLOW, "cell buffer holds %u records, tree has %u",
                         cell_capacity, ncell);
    const size_t cells_bytes = cells ? sizeof(GpuCell) * (size_t)ncell : 0;
    const size_t bodies_bytes = bodies ? sizeof(GpuBody) * (size_t)sn : 0;
    const size_t entries_bytes = entries ? sizeof(GpuEntry) * (size_t)sn : 0;
    if (cells_bytes + bodies_bytes + entries_bytes == 0) return BH_OK;
    PoolBlock block(dev);
    cudaError_t e = block.get(cells_bytes + bodies_bytes + entries_bytes);
    GpuCell* d_c = reinterpret_cast<GpuCell*>(block.at);
    GpuBody* d_b = reinterpret_cast<GpuBody*>(block.at + cells_bytes);
    GpuEntry* d_e = reinterpret_cast<GpuEntry*>(block.at + cells_bytes + bodies_bytes);
    if (!e)
        e = launch_export(b->bb, 0, entries_bytes ? d_e : nullptr, bodies_bytes ? d_b : nullptr,
                          cells_bytes ? d_c : nullptr, s);
    if (!e && entries_bytes) e = copy_down(dev, entries, d_e, entries_bytes);
    if (!e && bodies_bytes) e = copy_down(dev, bodies, d_b, bodies_bytes);
    if (!e && cells_bytes) e = copy_down(dev, cells, d_c, cells_bytes);
    if (!e) e = block.wait();
    if (e) return cuda_fail(e, "tree evidence");
    return BH_OK;
}

extern "C" int galaxy_bh_tree_footprint(uint32_t n, const bh_config* cfg, uint64_t* bytes) {
    if (!cfg || !bytes) return set_error(BH_INVALID_ARG, "null argument");
    int rc = validate_config(cfg);
    if (rc) return rc;
    const uint32_t counts[1] = {n};
    Layout L = plan_layout(counts, cfg, 1);
    *bytes = plan_arena(L, 1).total();
    return BH_OK;
}

extern "C" int galaxy_bh_tree_buffer_bytes(bh_tree* tree, uint64_t* bytes) {
    if (!tree || !bytes) return set_error(BH_INVALID_ARG, "null argument");
    *bytes = tree->batch->arena_bytes;
    return BH_OK;
}

extern "C" int galaxy_bh_step(bh_device* dev, bh_state* st, bh_tree* tree, const bh_config* cfg,
                              double dt, uint32_t nsteps) {
    int rc = tree_check(dev, st, tree);
    if (rc) return rc;
    if (!tree->built) return set_error(BH_INVALID_ARG, "step requires rebuild + force first");
    float f = 0.f;
    if ((rc = checked_dt(dt, &f))) return rc;
    if (nsteps == 0) return BH_OK;
    tree->batch->h_sims[0].dt = f;
    if ((rc = apply_configs(tree->batch, cfg, true))) return rc;
    tree->batch->built_theta = cfg->theta;
    tree->batch->built_g = cfg->g;
    rc = run_graphs(tree->batch, nsteps);
    tree->built = rc == BH_OK;
    return rc;
}

// ----------------------------------------------------------- packed (2B1) --

static int packed_checks(const BhSettings* settings, const GpuBody* bodies, uint32_t n,
                         const GpuEntry* entries, const GpuCell* cells, uint32_t cell_count) {
    if (!settings || !bodies || !entries || !cells)
        return set_error(BH_INVALID_ARG, "null argument");
    if (n == 0 || cell_count == 0)
        return set_error(BH_INVALID_ARG, "Barnes-Hut bodies/cells requires a non-empty buffer");
    if (settings->info[0] != n) return set_error(BH_INVALID_ARG, "flat tree/body cardinality mismatch");
    if (settings->info[2] >= cell_count) return set_error(BH_INVALID_ARG, "flat tree has invalid root");
    return BH_OK;
}

// Uploads the packed records and walks them; d_out: the accelerations, or null
// to keep them in the call's own block and copy them to `out`.
static int run_packed(bh_device* dev, const BhSettings* settings, const GpuBody* bodies,
                      uint32_t n, const GpuEntry* entries, const GpuCell* cells,
                      uint32_t cell_count, float4* d_out, GpuAccel* out,
                      bh_stage_timing* timing) {
    cudaStream_t s = dev->stream;
    const size_t body_bytes = sizeof(GpuBody) * (size_t)n, entry_bytes = sizeof(GpuEntry) * (size_t)n;
    const size_t cell_bytes = sizeof(GpuCell) * (size_t)cell_count;
    const size_t out_bytes = d_out ? 0 : sizeof(float4) * (size_t)n;
    PoolBlock block(dev);
    // cells, bodies, settings (32 bytes), entries, accelerations, the walk's two
    // error words and the first non-finite result
    CK(block.get(cell_bytes + body_bytes + sizeof(BhSettings) + entry_bytes + out_bytes + 16),
       "packed traversal allocation");
    GpuCell* d_c = reinterpret_cast<GpuCell*>(block.at);
    GpuBody* d_b = reinterpret_cast<GpuBody*>(block.at + cell_bytes);
    BhSettings* d_s = reinterpret_cast<BhSettings*>((char*)d_b + body_bytes);
    GpuEntry* d_e = reinterpret_cast<GpuEntry*>(d_s + 1);
    char* rest = (char*)d_e + entry_bytes;
    if (!d_out) {
        d_out = reinterpret_cast<float4*>(rest);
        CK(cudaMemsetAsync(d_out, 0, out_bytes, s), "memset");
    }
    uint32_t* d_err = reinterpret_cast<uint32_t*>(rest + out_bytes);
    uint32_t err[3] = {0, 0, kNone};
    cudaEventRecord(dev->ev[0], s);
    cudaError_t e = cudaSuccess;
    if ((e = cudaMemcpyAsync(d_s, settings, sizeof(BhSettings), cudaMemcpyHostToDevice, s)) ||
        (e = copy_up(dev, d_b, bodies, body_bytes)) || (e = copy_up(dev, d_e, entries, entry_bytes)) ||
        (e = copy_up(dev, d_c, cells, cell_bytes)) || (e = cudaMemsetAsync(d_err, 0, 8, s)) ||
        (e = cudaMemsetAsync(d_err + 2, 0xff, 4, s)))
        return cuda_fail(e, "packed traversal");
    cudaEventRecord(dev->ev[1], s);
    if ((e = launch_traverse_packed(d_s, d_b, d_e, d_c, n, cell_count, d_out, d_err, s)))
        return cuda_fail(e, "packed traversal");
    cudaEventRecord(dev->ev[2], s);
    if (out && (e = launch_check_records(d_out, 1, n, d_err + 2, s)))
        return cuda_fail(e, "packed traversal");
    // the error words first: a walk that failed leaves the caller's array alone
    if ((e = cudaMemcpyAsync(err, d_err, sizeof err, cudaMemcpyDeviceToHost, s)) ||
        (e = block.wait()))
        return cuda_fail(e, "packed traversal");
    float up = 0.f, walk = 0.f, down = 0.f;
    if (out && !err[0]) {
        block.idle = false;
        cudaEventRecord(dev->ev[3], s);
        if ((e = copy_down(dev, out, d_out, out_bytes))) return cuda_fail(e, "acceleration readback");
        cudaEventRecord(dev->ev[4], s);
        if ((e = block.wait())) return cuda_fail(e, "acceleration readback");
        cudaEventElapsedTime(&down, dev->ev[3], dev->ev[4]);
    }
    if (timing) {
        cudaEventElapsedTime(&up, dev->ev[0], dev->ev[1]);
        cudaEventElapsedTime(&walk, dev->ev[1], dev->ev[2]);
        *timing = bh_stage_timing{up * 1e-3, walk * 1e-3, down * 1e-3};
    }
    if (err[0] & kErrPackedStack)
        return set_error(BH_CAPACITY_OVERFLOW, "packed traversal stack exceeded 64 entries");
    if (err[0]) return set_error(BH_INVALID_ARG, "packed tree holds an out-of-range index");
    if (out && err[2] != kNone)
        return set_error(BH_NONFINITE, "GPU produced non-finite acceleration for body %u", err[2]);
    return BH_OK;
}

extern "C" int galaxy_bh_traverse_packed(bh_device* dev, const BhSettings* settings,
                                         const GpuBody* bodies, uint32_t n,
                                         const GpuEntry* entries, const GpuCell* cells,
                                         uint32_t cell_count, GpuAccel* out,
                                         bh_stage_timing* timing) {
    int rc = enter(dev);
    if (rc) return rc;
    if (!out) return set_error(BH_INVALID_ARG, "null argument");
    if ((rc = packed_checks(settings, bodies, n, entries, cells, cell_count))) return rc;
    return run_packed(dev, settings, bodies, n, entries, cells, cell_count, nullptr, out, timing);
}

extern "C" int galaxy_bh_force_into(bh_device* dev, bh_state* st, const BhSettings* settings,
                                    const GpuBody* bodies, const GpuEntry* entries,
                                    const GpuCell* cells, uint32_t cell_count,
                                    bh_stage_timing* timing) {
    int rc = enter(dev);
    if (rc) return rc;
    if (!st) return set_error(BH_INVALID_ARG, "null state");
    if ((rc = packed_checks(settings, bodies, st->n, entries, cells, cell_count)))
        return set_error(rc, "Barnes-Hut force/tree count does not match evolving state");
    return run_packed(dev, settings, bodies, st->n, entries, cells, cell_count, st->d_accel, nullptr,
                      timing);
}

// ------------------------------------------------------------ batch API ----

struct bh_batch {
    bh_device* dev = nullptr;
    Batch* batch = nullptr;
    bool solved = false;
};

extern "C" int galaxy_bh_batch_create(bh_device* dev, bh_state* const* states,
                                      const bh_config* cfgs, uint32_t count, bh_batch** out) {
    int rc = enter(dev);
    if (rc) return rc;
    if (!states || !cfgs || !out) return set_error(BH_INVALID_ARG, "null argument");
    *out = nullptr;
    for (uint32_t s = 0; s < count; ++s)
        if (cfgs[s].flags & BH_FLAG_POTENTIAL) {
            if (!states[s]) return set_error(BH_INVALID_ARG, "null state %u", s);
            if ((rc = ensure_potential(states[s]))) return rc;
        }
    Batch* b = nullptr;
    if ((rc = batch_build(dev, states, cfgs, count, &b))) return rc;
    bh_batch* h = new bh_batch();
    h->dev = dev;
    device_ref(dev);
    h->batch = b;
    *out = h;
    return BH_OK;
}

extern "C" int galaxy_bh_batch_destroy(bh_batch* batch) {
    if (!batch) return BH_OK;
    cudaSetDevice(batch->dev->ordinal);
    cudaStreamSynchronize(batch->dev->stream);
    delete batch->batch;
    bh_device* dev = batch->dev;
    delete batch;
    device_unref(dev);
    return BH_OK;
}

// Re-forms *batch over `count` states (creating it when null, destroying it
// when count is 0), keeping its arena when that is large enough: a serving
// loop's joins and leaves then allocate nothing once the arena has grown to
// the largest active set.
int gbh::batch_reform(bh_device* dev, bh_batch** batch, bh_state* const* states,
                      const bh_config* cfgs, uint32_t count) {
    if (!batch) return set_error(BH_INVALID_ARG, "null argument");
    if (count == 0) {
        galaxy_bh_batch_destroy(*batch);
        *batch = nullptr;
        return BH_OK;
    }
    if (!*batch) return galaxy_bh_batch_create(dev, states, cfgs, count, batch);
    int rc = enter(dev);
    if (rc) return rc;
    bh_batch* h = *batch;
    if (h->dev != dev) return set_error(BH_INVALID_ARG, "batch belongs to another device handle");
    if (!states || !cfgs) return set_error(BH_INVALID_ARG, "null argument");
    for (uint32_t s = 0; s < count; ++s)
        if (cfgs[s].flags & BH_FLAG_POTENTIAL) {
            if (!states[s]) return set_error(BH_INVALID_ARG, "null state %u", s);
            if ((rc = ensure_potential(states[s]))) return rc;
        }
    Batch* b = nullptr;
    Batch* donor = h->batch;
    h->batch = nullptr;
    h->solved = false;
    if ((rc = batch_build(dev, states, cfgs, count, &b, donor))) {
        galaxy_bh_batch_destroy(h);
        *batch = nullptr;
        return rc;
    }
    h->batch = b;
    return BH_OK;
}

extern "C" int galaxy_bh_batch_solve(bh_device* dev, bh_batch* batch) {
    int rc = enter(dev);
    if (rc) return rc;
    if (!batch || batch->dev != dev) return set_error(BH_INVALID_ARG, "batch does not belong to device");
    Batch* b = batch->batch;
    if ((rc = upload_sims(b))) return rc;
    if ((rc = enqueue_rebuild(b, 0, nullptr))) return rc;
    if ((rc = enqueue_force(b, false))) return rc;
    batch->solved = true;
    return check_device_errors(b);
}

extern "C" int galaxy_bh_batch_step(bh_device* dev, bh_batch* batch, const double* dts,
                                    uint32_t nsteps) {
    int rc = enter(dev);
    if (rc) return rc;
    if (!batch || !dts || batch->dev != dev) return set_error(BH_INVALID_ARG, "null argument");
    // Each member's acceleration buffer must already hold its boundary
    // acceleration (from galaxy_bh_batch_solve, galaxy_bh_force, or earlier
    // steps of any batch or tree): a batch re-formed after members left can
    // step at once.
    Batch* b = batch->batch;
    for (size_t s = 0; s < b->h_sims.size(); ++s) {
        float f = 0.f;
        if ((rc = checked_dt(dts[s], &f))) return rc;
        b->h_sims[s].dt = f;
    }
    if (nsteps == 0) return BH_OK;
    if ((rc = upload_sims(b))) return rc;
    return run_graphs(b, nsteps);
}

// Installs launch-shape knobs; the next step re-captures its graphs.
static int apply_tuning(Batch* b, const bh_tuning* t) {
    if (!t) return set_error(BH_INVALID_ARG, "null argument");
    if (t->radix_bits != 4 && t->radix_bits != 8)
        return set_error(BH_INVALID_ARG, "radix_bits must be 4 or 8, got %u", t->radix_bits);
    if (t->traverse_warps != 2 && t->traverse_warps != 4 && t->traverse_warps != 8)
        return set_error(BH_INVALID_ARG, "traverse_warps must be 2, 4 or 8, got %u",
                         t->traverse_warps);
    if (t->radix_bits != b->bb.radix_bits || t->traverse_warps != b->bb.trav_warps) {
        b->bb.radix_bits = t->radix_bits;
        b->bb.trav_warps = t->traverse_warps;
        b->graph_flags = 0xffffffffu;  // graphs hold the old launch shapes
    }
    return BH_OK;
}

extern "C" int galaxy_bh_batch_tune(bh_batch* batch, const bh_tuning* tuning) {
    if (!batch) return set_error(BH_INVALID_ARG, "null batch");
    return apply_tuning(batch->batch, tuning);
}

extern "C" int galaxy_bh_tree_tune(bh_tree* tree, const bh_tuning* tuning) {
    if (!tree) return set_error(BH_INVALID_ARG, "null tree");
    return apply_tuning(tree->batch, tuning);
}

extern "C" int galaxy_bh_batch_bytes(bh_batch* batch, uint64_t* bytes) {
    if (!batch || !bytes) return set_error(BH_INVALID_ARG, "null argument");
    *bytes = batch->batch->arena_bytes;
    return BH_OK;
}
