// SPDX-License-Identifier: Apache-2.0
//
// sm_100a kernels of the Barnes-Hut evolution step.  Every kernel covers all
// simulations of a batch in one launch (the plain path is a batch of one):
//
//   k_integrate   kick/drift/final-kick (runtime/src/nbody_evolve.wgsl) fused
//                 with the per-simulation f32 min/max bounds reduction
//   k_morton      f64 root bounds + 16-bit/axis quantization + Morton code
//                 (nbody/src/lib.rs:137-154, nbody/src/flat.rs:67-94), fused
//                 with the four 8-bit digit histograms of the radix sort
//   k_radix_pass  one stable LSD pass (onesweep: look-back by tile groups, warp
//                 match ranking, shared-memory staged scatter); the last pass
//                 also gathers the bodies into Morton order
//   k_sort_small  all of these and the chain scan of a simulation of at most
//                 65,536 bodies in one block or cluster
//   k_count_scan  cells per position + exclusive scan (cell numbering in the
//                 reference's recursive preorder, nbody/src/flat.rs:127-177)
//   k_aggregate   ranges, children, skip pointers of every cell and bottom-up
//                 f64 mass / centre of mass, identical arithmetic and order to
//                 nbody/src/flat.rs:179-215, in blocks of about 256 positions;
//                 k_aggregate_inner and _outer the cells across blocks
//   k_traverse    lane-parallel theta-MAC walk over node groups with per-warp
//                 interaction lists (nbody/src/flat.rs:270-346 decisions per
//                 body), f32 forces, exact f64 MAC in the guard band
//
// The f64 expressions that must reproduce the reference bit for bit use the
// explicit round-to-nearest intrinsics (__dadd_rn, __dmul_rn, ...), which
// nvcc never contracts into FMAs.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "bh_internal.cuh"

namespace gbh {

namespace {

constexpr unsigned kFull = 0xffffffffu;

#ifndef GBH_PDL
#define GBH_PDL 1
#endif

// Launches a kernel of the step with programmatic stream serialization, so
// its launch overlaps the previous kernel's tail (see wait_for_predecessor).
template <typename... KArgs, typename... Args>
static cudaError_t launch_clusters(void (*kernel)(KArgs...), uint32_t cluster, dim3 grid,
                                   dim3 block, size_t smem, cudaStream_t s, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = GBH_PDL;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

template <typename... KArgs, typename... Args>
static cudaError_t launch_step(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem,
                               cudaStream_t s, Args... args) {
    return launch_clusters(kernel, 1, grid, block, smem, s, args...);
}

__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31u; }

__device__ __forceinline__ void set_err(uint32_t* err, uint32_t bits) { atomicOr(err, bits); }

// Programmatic dependent launch: a kernel of the step may be launched while
// its predecessor drains; it waits here, before touching any memory, until
// the predecessor has completed and its writes are visible (a no-op for a
// launch without the attribute).
__device__ __forceinline__ void wait_for_predecessor() {
#if GBH_PDL
    asm volatile("griddepcontrol.wait;" ::: "memory");
#endif
}

// Whether a wait of the step ran out.  The codes may be unsorted then and the
// chains' sums short, and what the sort's passes and the aggregates read and write
// by them could lie outside their arrays.
__device__ __forceinline__ bool gave_up(const uint32_t* err) {
    return (*err & kErrLookbackTimeout) != 0u;
}

// Order-preserving float <-> uint mapping (for integer atomics on floats).
__device__ __forceinline__ uint32_t enc_f32(float f) {
    uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float dec_f32(uint32_t e) {
    uint32_t u = (e & 0x80000000u) ? (e & 0x7fffffffu) : ~e;
    return __uint_as_float(u);
}

struct RootBounds {
    double cx, cy, half;
};

// nbody/src/lib.rs:137-154 over the f32 min/max promoted to f64.
__device__ __forceinline__ RootBounds root_bounds(float mnx, float mny, float mxx, float mxy) {
    const double min_x = mnx, min_y = mny, max_x = mxx, max_y = mxy;
    double span = fmax(fmax(__dsub_rn(max_x, min_x), __dsub_rn(max_y, min_y)), 1e-12);
    RootBounds r;
    r.cx = __dmul_rn(__dadd_rn(min_x, max_x), 0.5);
    r.cy = __dmul_rn(__dadd_rn(min_y, max_y), 0.5);
    r.half = __dadd_rn(__dmul_rn(span, 0.500000000001), 1e-12);
    return r;
}

__device__ __forceinline__ RootBounds root_bounds_from(const uint32_t* mm) {
    return root_bounds(dec_f32(~mm[0]), dec_f32(~mm[1]), dec_f32(mm[2]), dec_f32(mm[3]));
}

// Root width / theta, +inf at theta = 0 (every cell opens).
__device__ __forceinline__ double crit_of(double root_half, double theta) {
    return theta > 0.0 ? __dmul_rn(root_half, 2.0) / theta : INFINITY;
}

// nbody/src/flat.rs:82-87
__device__ __forceinline__ uint32_t quantize_axis(double value, double center, double half) {
    double low = __dsub_rn(center, half);
    double width = __dmul_rn(half, 2.0);
    double scaled = floor(__dmul_rn(__ddiv_rn(__dsub_rn(value, low), width), 65536.0));
    scaled = fmin(fmax(scaled, 0.0), 65535.0);
    return (uint32_t)scaled;
}

// nbody/src/flat.rs:67-80
__device__ __forceinline__ uint32_t spread16(uint32_t v) {
    v &= 0x0000ffffu;
    v = (v | (v << 8)) & 0x00ff00ffu;
    v = (v | (v << 4)) & 0x0f0f0f0fu;
    v = (v | (v << 2)) & 0x33333333u;
    v = (v | (v << 1)) & 0x55555555u;
    return v;
}
__device__ __forceinline__ uint32_t morton2(uint32_t x, uint32_t y) {
    return spread16(x) | (spread16(y) << 1);
}

// Number of leading quadtree levels (2 bits each) two codes share; 16 when equal.
__device__ __forceinline__ uint32_t shared_levels(uint32_t a, uint32_t b) {
    return a == b ? 16u : ((uint32_t)__clz(a ^ b) >> 1);
}

// 2^-d as an exact double.
__device__ __forceinline__ double pow2_neg(uint32_t d) {
    return __longlong_as_double((long long)(1023 - (int)d) << 52);
}

// First index in [lo, hi) whose code is >= x (codes ascending there; hi if
// none), for NT targets at once, by 8-way partition: each round loads seven
// evenly spaced codes per unfinished target — all of them one round trip —
// and keeps the eighth of the range that holds the bound; the last <= 8
// positions are counted with independent loads.  A range of D positions
// takes log8(D) + 1 round trips instead of the ~2 log2(D) dependent loads of
// a binary search, which is what the few cells spanning most of the
// positions (near the root) wait for.
template <int NT>
__device__ __forceinline__ void kary_lower_bound(const uint32_t* codes, uint32_t lo, uint32_t hi,
                                                 const uint32_t (&x)[NT], uint32_t (&out)[NT]) {
    uint32_t l[NT], h[NT];
#pragma unroll
    for (int t = 0; t < NT; ++t) {
        l[t] = lo;
        h[t] = hi;
    }
    while (true) {
        bool more = false;
#pragma unroll
        for (int t = 0; t < NT; ++t) more = more || h[t] - l[t] > 8u;
        if (!more) break;
        uint32_t c[NT][7];
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            const uint32_t step = (h[t] - l[t]) / 8u;
#pragma unroll
            for (int j = 0; j < 7; ++j)
                c[t][j] = step ? __ldg(codes + l[t] + step * (uint32_t)(j + 1)) : 0u;
        }
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            const uint32_t step = (h[t] - l[t]) / 8u;
            if (!step) continue;
            uint32_t below = 0;  // probes below x: the probes are ascending
#pragma unroll
            for (int j = 0; j < 7; ++j) below += c[t][j] < x[t] ? 1u : 0u;
            const uint32_t nl = below ? l[t] + step * below + 1u : l[t];
            const uint32_t nh = below < 7u ? l[t] + step * (below + 1u) : h[t];
            l[t] = nl;
            h[t] = nh;
        }
    }
#pragma unroll
    for (int t = 0; t < NT; ++t) {
        uint32_t below = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j)
            below += (l[t] + (uint32_t)j < h[t] && __ldg(codes + l[t] + j) < x[t]) ? 1u : 0u;
        out[t] = l[t] + below;
    }
}

// Exclusive scan over a 256-thread block; *total gets the block sum.
__device__ __forceinline__ uint32_t block_exclusive_scan_256(uint32_t v, uint32_t* total,
                                                             uint32_t* smem8) {
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(kFull, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31) smem8[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < 8 ? smem8[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            uint32_t y = __shfl_up_sync(kFull, w, o);
            if (lane >= (uint32_t)o) w += y;
        }
        if (lane < 8) smem8[lane] = w;
    }
    __syncthreads();
    uint32_t wp = warp ? smem8[warp - 1] : 0u;
    *total = smem8[7];
    __syncthreads();
    return wp + x - v;
}

__device__ __forceinline__ uint32_t ld_volatile(const uint32_t* p) {
    return *(const volatile uint32_t*)p;
}
__device__ __forceinline__ unsigned long long ld_volatile64(const unsigned long long* p) {
    return *(const volatile unsigned long long*)p;
}

// Bounded wait budget for look-back spins (~1 s at 2 GHz).
constexpr long long kSpinCycles = 2000000000ll;

}  // namespace

// ============================================================ integrate ====

// runtime/src/nbody_evolve.wgsl:19-46 with explicit f32 roundings (no FMA):
// half_velocity = v + (0.5*dt)*a ; x = x + dt*half_velocity.  Mode 3 runs the
// final kick of one step and the kick-drift of the next with the same two
// roundings as two separate launches.  Modes 0, 1, 3 also reduce the
// per-simulation f32 bounds of the (new) positions.
#ifndef GBH_INTEGRATE_UNROLL
#define GBH_INTEGRATE_UNROLL 4
#endif
// chunks whose loads a warp keeps in flight (modes with the bounds reduction)
constexpr int kIntegrateUnrollBounds = GBH_INTEGRATE_UNROLL;

// The kick / drift of one record.
__device__ __forceinline__ void integrate(int mode, float dt, float4& pm, float4& v,
                                          const float4& a) {
    const float hdt = __fmul_rn(0.5f, dt);
    if (mode == 2 || mode == 3) {
        v.x = __fadd_rn(v.x, __fmul_rn(hdt, a.x));
        v.y = __fadd_rn(v.y, __fmul_rn(hdt, a.y));
    }
    if (mode == 1 || mode == 3) {
        v.x = __fadd_rn(v.x, __fmul_rn(hdt, a.x));
        v.y = __fadd_rn(v.y, __fmul_rn(hdt, a.y));
        pm.x = __fadd_rn(pm.x, __fmul_rn(dt, v.x));
        pm.y = __fadd_rn(pm.y, __fmul_rn(dt, v.y));
    }
}

template <int MODE>
__global__ void __launch_bounds__(256) k_integrate(const SimDesc* __restrict__ sims,
                                                   const uint32_t* __restrict__ chunk_sim,
                                                   uint32_t nchunks, uint32_t* minmax) {
    wait_for_predecessor();
    constexpr bool kBounds = MODE != 2;
    // without the bounds reduction (no atomics) one warp per chunk streams
    // best; with it, fewer blocks each keeping several chunks' loads in flight
    constexpr int kIntegrateUnroll = kBounds ? kIntegrateUnrollBounds : 1;
    __shared__ uint32_t s_sim[8];
    __shared__ float s_val[8][4];
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    // grid-stride over chunks, kIntegrateUnroll strides per round: at any
    // moment the warps of the grid stream one contiguous region
    const uint32_t nwarps = gridDim.x * 8;
    const uint32_t gw = blockIdx.x * 8 + warp;
    uint32_t cur = kNone;
    // fields of simulation `cur`, reloaded only when the simulation changes
    GpuEvolveState* st = nullptr;
    const float4* acc = nullptr;
    uint32_t off = 0, n = 0;
    float dt = 0.f;
    float mnx = INFINITY, mny = INFINITY, mxx = -INFINITY, mxy = -INFINITY;

    auto warp_reduce = [&]() {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            mnx = fminf(mnx, __shfl_xor_sync(kFull, mnx, o));
            mny = fminf(mny, __shfl_xor_sync(kFull, mny, o));
            mxx = fmaxf(mxx, __shfl_xor_sync(kFull, mxx, o));
            mxy = fmaxf(mxy, __shfl_xor_sync(kFull, mxy, o));
        }
    };
    // warp-uniform: publishes the bounds of the previous simulation
    auto enter_sim = [&](uint32_t s) {
        if (s == cur) return;
        if (kBounds && cur != kNone) {
            warp_reduce();
            if (lane == 0) {
                atomicMax(&minmax[4 * cur + 0], ~enc_f32(mnx));
                atomicMax(&minmax[4 * cur + 1], ~enc_f32(mny));
                atomicMax(&minmax[4 * cur + 2], enc_f32(mxx));
                atomicMax(&minmax[4 * cur + 3], enc_f32(mxy));
            }
            mnx = mny = INFINITY;
            mxx = mxy = -INFINITY;
        }
        cur = s;
        const SimDesc& sd = sims[s];
        st = sd.state;
        acc = sd.accel;
        off = sd.off;
        n = sd.n;
        dt = sd.dt;
    };
    auto update = [&](float4& pm, float4& v, const float4& a) { integrate(MODE, dt, pm, v, a); };
    auto bound = [&](const float4& pm) {
        if (kBounds) {
            mnx = fminf(mnx, pm.x);
            mny = fminf(mny, pm.y);
            mxx = fmaxf(mxx, pm.x);
            mxy = fmaxf(mxy, pm.y);
        }
    };
    auto one_chunk = [&](uint32_t chunk, uint32_t s) {
        if (s == kNone) return;
        enter_sim(s);
        const uint32_t i = chunk * kChunk + lane - off;
        if (i >= n) return;
        float4* rec = reinterpret_cast<float4*>(st + i);
        float4 pm = rec[0];
        if (MODE != 0) {
            float4 v = rec[1];
            update(pm, v, acc[i]);
            if (MODE != 2) rec[0] = pm;
            rec[1] = v;
        }
        bound(pm);
    };

    constexpr uint32_t kPast = kNone - 1u;  // a slot past the last chunk
    for (uint32_t round = gw; round < nchunks; round += kIntegrateUnroll * nwarps) {
        uint32_t sv[kIntegrateUnroll], cv[kIntegrateUnroll];
#pragma unroll
        for (int j = 0; j < kIntegrateUnroll; ++j) {
            cv[j] = round + (uint32_t)j * nwarps;
            sv[j] = cv[j] < nchunks ? chunk_sim[cv[j]] : kPast;
        }
        bool same = sv[0] != kNone;
#pragma unroll
        for (int j = 1; j < kIntegrateUnroll; ++j) same = same && (sv[j] == sv[0] || sv[j] == kPast);
        if (!same) {
#pragma unroll 1
            for (int j = 0; j < kIntegrateUnroll; ++j)
                if (sv[j] != kPast) one_chunk(cv[j], sv[j]);
            continue;
        }
        // one simulation: every load of the run first, then the updates
        enter_sim(sv[0]);
        float4 pm[kIntegrateUnroll], v[kIntegrateUnroll], a[kIntegrateUnroll];
        bool ok[kIntegrateUnroll];
#pragma unroll
        for (int j = 0; j < kIntegrateUnroll; ++j) {
            const uint32_t i = cv[j] * kChunk + lane - off;
            ok[j] = sv[j] != kPast && i < n;
            if (ok[j]) {
                const float4* rec = reinterpret_cast<const float4*>(st + i);
                pm[j] = rec[0];
                if (MODE != 0) {
                    v[j] = rec[1];
                    a[j] = acc[i];
                }
            }
        }
#pragma unroll
        for (int j = 0; j < kIntegrateUnroll; ++j) {
            if (!ok[j]) continue;
            const uint32_t i = cv[j] * kChunk + lane - off;
            if (MODE != 0) {
                update(pm[j], v[j], a[j]);
                float4* rec = reinterpret_cast<float4*>(st + i);
                if (MODE != 2) rec[0] = pm[j];
                rec[1] = v[j];
            }
            bound(pm[j]);
        }
    }
    if (!kBounds) return;
    warp_reduce();
    if (lane == 0) {
        s_sim[warp] = cur;
        s_val[warp][0] = mnx;
        s_val[warp][1] = mny;
        s_val[warp][2] = mxx;
        s_val[warp][3] = mxy;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t run = kNone;
        float a0 = 0, a1 = 0, a2 = 0, a3 = 0;
        for (int w = 0; w <= 8; ++w) {
            const uint32_t sw = w < 8 ? s_sim[w] : kNone;
            if (w == 8 || sw != run) {
                if (run != kNone) {
                    atomicMax(&minmax[4 * run + 0], ~enc_f32(a0));
                    atomicMax(&minmax[4 * run + 1], ~enc_f32(a1));
                    atomicMax(&minmax[4 * run + 2], enc_f32(a2));
                    atomicMax(&minmax[4 * run + 3], enc_f32(a3));
                }
                if (w == 8) break;
                run = sw;
                a0 = s_val[w][0];
                a1 = s_val[w][1];
                a2 = s_val[w][2];
                a3 = s_val[w][3];
            } else {
                a0 = fminf(a0, s_val[w][0]);
                a1 = fminf(a1, s_val[w][1]);
                a2 = fmaxf(a2, s_val[w][2]);
                a3 = fmaxf(a3, s_val[w][3]);
            }
        }
    }
}

// ============================================================== morton ====

constexpr uint32_t kHistStride = kRadixPasses * kRadixDigits;  // histogram words per sim

// One block per radix tile: Morton codes of the tile's bodies (resident
// order) plus the tile's contribution to the digit histograms of every pass
// of a BITS-wide LSD sort (hist[sim][pass * 2^BITS + digit]).
// Threads per Morton block (one radix tile of kTile keys): 512 hide more of
// the quantization's f64 latency than 256 (and than 1024).
constexpr int kMortonThreads = 512;
constexpr int kMortonItems = (int)kTile / kMortonThreads;
static_assert(kMortonItems * kMortonThreads == (int)kTile, "a Morton block covers one tile");

template <int BITS>
__global__ void __launch_bounds__(kMortonThreads) k_morton(const SimDesc* __restrict__ sims,
                                                         const Tile* __restrict__ tiles,
                                                         const uint32_t* __restrict__ minmax,
                                                         uint32_t* __restrict__ keys,
                                                         uint32_t* hist, uint32_t* group_words,
                                                         SimOut* simout) {
    wait_for_predecessor();
    constexpr int kPasses = 32 / BITS;
    constexpr uint32_t kDig = 1u << BITS;
    __shared__ uint32_t sh[kPasses * kDig];
    for (int k = threadIdx.x; k < kPasses * (int)kDig; k += kMortonThreads) sh[k] = 0;
    __syncthreads();
    const Tile t = tiles[blockIdx.x];
    const SimDesc& sd = sims[t.sim];
    if (t.group != kNone && (t.start - sd.off) / kTile % kGroupTiles == 0u)
        for (uint32_t k = threadIdx.x; k < kGroupStride; k += kMortonThreads)
            group_words[(size_t)t.group * kGroupStride + k] = 0u;
    const RootBounds rb = root_bounds_from(minmax + 4 * t.sim);
    if (threadIdx.x == 0 && t.start == sd.off) {
        simout[t.sim].cx = rb.cx;
        simout[t.sim].cy = rb.cy;
        simout[t.sim].half = rb.half;
        simout[t.sim].crit0 = crit_of(rb.half, sd.theta);
    }
#pragma unroll
    for (int k = 0; k < kMortonItems; ++k) {
        const uint32_t idx = k * kMortonThreads + threadIdx.x;
        if (idx < t.count) {
            const uint32_t p = t.start + idx;
            const float2 xy = *reinterpret_cast<const float2*>(sd.state + (p - sd.off));
            const uint32_t code = morton2(quantize_axis((double)xy.x, rb.cx, rb.half),
                                          quantize_axis((double)xy.y, rb.cy, rb.half));
            keys[p] = code;
#pragma unroll
            for (int pass = 0; pass < kPasses; ++pass)
                atomicAdd(&sh[pass * kDig + ((code >> (BITS * pass)) & (kDig - 1u))], 1u);
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < kPasses * (int)kDig; k += kMortonThreads) {
        const uint32_t c = sh[k];
        if (c) atomicAdd(&hist[(size_t)t.sim * kHistStride + k], c);
    }
}

// ============================================================== radix =====

#ifndef GBH_LOOK_WINDOW
#define GBH_LOOK_WINDOW 16
#endif
constexpr int kLookWindow = GBH_LOOK_WINDOW;  // counts loaded per look-back round trip
// A published count: kGroupTiles << kCountBits | count.  A tile's word gets it at
// once; its group's word, to which each of the kGroupTiles tiles adds 1 <<
// kCountBits | count, once they all have.
constexpr uint32_t kCountBits = 20;
constexpr uint32_t kCountMask = (1u << kCountBits) - 1u;
static_assert(kGroupTiles * kTile <= kCountMask, "a group's count fits its bits");
constexpr uint32_t kPrefix = 1u << 31;  // marks a published prefix

// Look-back for one digit: the counts of the `tiles` tiles of the group before
// this one (tile_words[i * stride]), then of the `groups` groups before it, the
// nearest first (group_words[-i * kGroupStride], i from 1), up to the first whose
// last tile has published the sum through it (kPrefix | sum, kGroupWords further).
// kLookWindow loads per round trip, polled until they are published.  The wait is
// bounded: once `limit` clock cycles have passed since it began and a count is
// missing, it sets kErrLookbackTimeout and returns the sum so far, which is at most
// the true prefix (the caller's writes stay in range).
__device__ __forceinline__ uint32_t lookback_digit(const uint32_t* tile_words, uint32_t stride,
                                                   uint32_t tiles, const uint32_t* group_words,
                                                   uint32_t groups, uint32_t* err,
                                                   long long limit) {
    uint32_t excl = 0;
    const long long t0 = clock64();
    for (uint32_t i0 = 0; i0 < tiles; i0 += kLookWindow) {
        uint32_t sum;
        bool all;
        do {
            uint32_t f[kLookWindow];
#pragma unroll
            for (int j = 0; j < kLookWindow; ++j)
                f[j] = i0 + j < tiles ? ld_volatile(tile_words + (size_t)(i0 + j) * stride)
                                      : kGroupTiles << kCountBits;
            sum = 0;
            all = true;
#pragma unroll
            for (int j = 0; j < kLookWindow; ++j) {
                all = all && f[j] >> kCountBits == kGroupTiles;
                sum += f[j] & kCountMask;
            }
            if (!all && clock64() - t0 > limit) {
                set_err(err, kErrLookbackTimeout);
                return excl;
            }
        } while (!all);
        excl += sum;
    }
    constexpr int kGroupWindow = kLookWindow / 2;
    for (uint32_t i0 = 1; i0 <= groups;) {
        uint32_t f[kGroupWindow], prefix[kGroupWindow];
#pragma unroll
        for (int j = 0; j < kGroupWindow; ++j) {
            const uint32_t* at = group_words - (size_t)min(i0 + j, groups) * kGroupStride;
            f[j] = ld_volatile(at);
            prefix[j] = ld_volatile(at + kGroupWords);
        }
        bool ready = true, done = false;
        uint32_t used = 0;
#pragma unroll
        for (int j = 0; j < kGroupWindow; ++j) {
            if (done || !ready || i0 + j > groups) continue;
            done = (prefix[j] & kPrefix) != 0u;
            ready = done || f[j] >> kCountBits == kGroupTiles;
            if (ready) excl += done ? prefix[j] & ~kPrefix : f[j] & kCountMask;
            used += ready;
        }
        if (done) break;
        i0 += used;
        if (!ready && clock64() - t0 > limit) {
            set_err(err, kErrLookbackTimeout);
            break;
        }
    }
    return excl;
}

// Failure-detection probe: the sort's look-back wait, one thread per digit, so
// every thread must give up after `limit` cycles and report the timeout.  Block 0
// waits as tile 1 of a simulation whose first tile never publishes, block 1 as the
// first tile of the third group, behind a group that has published a count of 1 a
// digit and one that never does.  words: zeros, kRadixDigits for the tile and
// kGroupStride for each group; err and out: a word, and kRadixDigits, a block.
__global__ void k_wait_probe(uint32_t* words, uint32_t* err, long long limit, uint32_t* out) {
    const uint32_t d = threadIdx.x;
    if (blockIdx.x == 0) {
        out[d] = lookback_digit(words + d, kRadixDigits, 1u, nullptr, 0u, err, limit);
    } else {
        uint32_t* group = words + kRadixDigits + 2u * kGroupStride + d;
        atomicExch(group - kGroupStride, kGroupTiles << kCountBits | 1u);
        out[kRadixDigits + d] = lookback_digit(nullptr, 0u, 0u, group, 2u, err + 1, limit);
    }
}

// One stable BITS-wide LSD pass (BITS = 8: 4 passes, 4: 8 passes) over every
// simulation's keys.  Tiles never cross simulations; within a simulation,
// tile order is key order and the look-back adds the digit counts of the
// preceding tiles.  Items are ranked warp by warp in key order (the
// lanes sharing a digit found with one ballot per digit bit), so equal
// digits keep their input order: the permutation equals a stable sort by
// code, as Rust's sort_by_key (nbody/src/flat.rs:233-234).
// A tile's counts go to its own words and, added, to those of its group of
// kGroupTiles tiles, so its look-back reads at most 31 tiles and the groups before
// it up to a known prefix, 16 words a round trip, where a chain of tiles advanced 8
// a round trip: 2^20 bodies' four passes 80 -> 74 us, 2^18 51 -> 47, 2^24 1,030 ->
// 935 (1,062 without the groups' prefixes, and 1.5 us less then at 2^20).  What is
// left, in cycles of a tile at 2^20 (2 tiles an SM): loads 2,500, ranking 4,000 to
// 5,000, waiting for the slowest of the tiles before it 5,000 to 9,000, scans and
// the local scatter 3,000, stores 2,000, and in the last pass the gather of a random
// 32-byte sector a body, 20,000 (with its loads issued together and no store of the
// values, which the bodies' records carry, 74 -> 71 us).  Counting with shared
// atomics before the ranking, to publish earlier, costs more than it saves (76 us;
// 2^18 57).
// MINB tiles share an SM: 2 (up to 128 registers) for sorts of one wave,
// 3 (80 registers) for sorts of many waves of tiles (large batches).
template <int BITS, int PASS, bool LAST, int MINB>
__global__ void __launch_bounds__(kSortThreads, MINB) k_radix_pass(
    const SimDesc* __restrict__ sims, const Tile* __restrict__ tiles, uint32_t* tile_counter,
    const uint32_t* __restrict__ hist, uint32_t* flags, uint32_t* group_words,
    const uint32_t* __restrict__ keys_in,
    const uint32_t* __restrict__ vals_in, uint32_t* __restrict__ keys_out,
    uint32_t* __restrict__ vals_out, float4* __restrict__ sbody, uint32_t* err) {
    wait_for_predecessor();
    constexpr uint32_t kDig = 1u << BITS;
    __shared__ uint32_t s_tile;
    __shared__ bool s_stop;
    __shared__ uint32_t s_whist[8][kDig];
    __shared__ uint32_t s_tprefix[kDig];
    __shared__ uint32_t s_out[kDig];
    __shared__ uint32_t s_keys[kTile];
    __shared__ uint32_t s_vals[kTile];
    __shared__ uint32_t s_scan[8];

    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        s_tile = atomicAdd(tile_counter, 1u);
        // in an earlier pass, or a tile of this one: read once, for the whole block
        s_stop = gave_up(err);
    }
    for (int k = threadIdx.x; k < 8 * (int)kDig; k += kSortThreads) (&s_whist[0][0])[k] = 0;
    __syncthreads();
    if (s_stop) return;
    const uint32_t t = s_tile;
    const Tile tl = tiles[t];
    const SimDesc& sd = sims[tl.sim];
    const uint32_t shift = (uint32_t)BITS * PASS;
    const uint32_t lt_mask = (1u << lane) - 1u;

    uint32_t key[kSortItems], val[kSortItems], rank[kSortItems];
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        const uint32_t idx = warp * (kSortItems * 32u) + r * 32u + lane;
        const bool valid = idx < tl.count;
        const uint32_t p = tl.start + idx;
        key[r] = valid ? keys_in[p] : 0u;
        val[r] = valid ? (PASS == 0 ? p - sd.off : vals_in[p]) : 0u;
    }
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        const uint32_t idx = warp * (kSortItems * 32u) + r * 32u + lane;
        const bool valid = idx < tl.count;
        const uint32_t d = (key[r] >> shift) & (kDig - 1u);
        // valid lanes holding the same digit: one ballot per digit bit
        uint32_t peers = __ballot_sync(kFull, valid);
#pragma unroll
        for (int bit = 0; bit < BITS; ++bit) {
            const uint32_t m = __ballot_sync(kFull, (d >> bit) & 1u);
            peers &= ((d >> bit) & 1u) ? m : ~m;
        }
        const uint32_t leader = __ffs(peers) - 1u;
        uint32_t b = 0;
        if (valid && lane == leader) {
            b = s_whist[warp][d];
            s_whist[warp][d] = b + __popc(peers);
        }
        b = __shfl_sync(kFull, b, leader);
        rank[r] = b + __popc(peers & lt_mask);
        __syncwarp();
    }
    __syncthreads();

    // Thread d < 2^BITS owns digit d: warp offsets, tile count, look-back,
    // bases (the other threads feed zeros to the block scans).
    const uint32_t d = threadIdx.x;
    const bool owner = d < kDig;
    uint32_t run = 0;
    if (owner) {
#pragma unroll
        for (int w = 0; w < 8; ++w) {
            const uint32_t c = s_whist[w][d];
            s_whist[w][d] = run;
            run += c;
        }
    }
    const uint32_t before = t - sd.first_tile, in_group = before % kGroupTiles;
    uint32_t excl = 0;
    if (owner && tl.group != kNone) {
        uint32_t* group = group_words + (size_t)tl.group * kGroupStride + PASS * kDig + d;
        atomicExch(flags + (size_t)t * kDig + d, kGroupTiles << kCountBits | run);
        atomicAdd(group, 1u << kCountBits | run);
        excl = lookback_digit(flags + (size_t)(t - in_group) * kDig + d, kDig, in_group,
                              group, before / kGroupTiles, err, kSpinCycles);
        if (in_group == kGroupTiles - 1u) atomicExch(group + kGroupWords, kPrefix | (excl + run));
    }
    uint32_t tot;
    const uint32_t h = owner ? hist[(size_t)tl.sim * kHistStride + PASS * kDig + d] : 0u;
    const uint32_t gex = block_exclusive_scan_256(h, &tot, s_scan);
    const uint32_t tex = block_exclusive_scan_256(run, &tot, s_scan);
    if (owner) {
        s_tprefix[d] = tex;
        s_out[d] = sd.off + gex + excl - tex;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        const uint32_t idx = warp * (kSortItems * 32u) + r * 32u + lane;
        if (idx < tl.count) {
            const uint32_t dg = (key[r] >> shift) & (kDig - 1u);
            const uint32_t slot = s_tprefix[dg] + s_whist[warp][dg] + rank[r];
            s_keys[slot] = key[r];
            s_vals[slot] = val[r];
        }
    }
    __syncthreads();
    // the gather's loads are issued four at a time
    constexpr int kGather = LAST ? 4 : 1;
#pragma unroll
    for (int k0 = 0; k0 < kSortItems; k0 += kGather) {
        float4 pm[kGather];
#pragma unroll
        for (int k = 0; LAST && k < kGather; ++k) {
            const uint32_t slot = (k0 + k) * kSortThreads + threadIdx.x;
            if (slot < tl.count)
                pm[k] = __ldcg(reinterpret_cast<const float4*>(sd.state + s_vals[slot]));
        }
#pragma unroll
        for (int k = 0; k < kGather; ++k) {
            const uint32_t slot = (k0 + k) * kSortThreads + threadIdx.x;
            if (slot < tl.count) {
                const uint32_t kk = s_keys[slot];
                const uint32_t vv = s_vals[slot];
                const uint32_t dest = s_out[(kk >> shift) & (kDig - 1u)] + slot;
                keys_out[dest] = kk;
                if (LAST)  // the values end in the bodies' records
                    sbody[dest] = make_float4(pm[k].x, pm[k].y, pm[k].z, __uint_as_float(vv));
                else
                    vals_out[dest] = vv;
            }
        }
    }
}

// ========================================================== count + scan ==

// Cells whose range starts at sorted position i (a "chain": depths
// d_min..D).  Cell (d, i) exists iff i starts a depth-d group and its parent
// group holds more than `bucket` bodies; it is internal iff it holds more
// than `bucket` bodies and d < max_depth (nbody/src/flat.rs:145).
template <typename Codes>
__device__ __forceinline__ uint32_t chain_count(const Codes sc, uint32_t i, uint32_t n,
                                                uint32_t bucket, uint32_t maxd,
                                                uint32_t* dmin_out) {
    const uint32_t ci = sc[i];
    const uint32_t dmin = i == 0 ? 0u : shared_levels(sc[i - 1], ci) + 1u;
    *dmin_out = dmin;
    if (dmin > maxd) return 0;
    if (i > 0 && bucket > 1) {
        // parent group (depth dmin-1) holds i-1 and i; needs > bucket bodies:
        // some window [j, j+bucket] containing both lies inside it.
        const uint32_t pd = dmin - 1u;
        const uint32_t jlo = i >= bucket ? i - bucket : 0u;
        bool ok = false;
        for (uint32_t j = jlo; j < i && j + bucket < n; ++j) {
            if (shared_levels(sc[j], sc[j + bucket]) >= pd) {
                ok = true;
                break;
            }
        }
        if (!ok) return 0;
    }
    const int lw = (i + bucket < n) ? (int)shared_levels(ci, sc[i + bucket]) : -1;
    const int deepest = max((int)dmin, min((int)maxd, lw + 1));
    return (uint32_t)(deepest - (int)dmin + 1);
}

// k_aggregate's blocks own [cut_b, cut_b+1): cut b is the first position of the
// kAggCutWindow ones from b * kAggPositions on that starts a group of the least
// depth, so that few cells, and only shallow ones, span two blocks.
#ifndef GBH_AGG_POSITIONS
#define GBH_AGG_POSITIONS 256
#endif
#ifndef GBH_AGG_CUT_WINDOW
#define GBH_AGG_CUT_WINDOW 128
#endif
constexpr uint32_t kAggPositions = GBH_AGG_POSITIONS;
constexpr uint32_t kAggCutWindow = GBH_AGG_CUT_WINDOW;
static_assert(kAggCutWindow == 32u * kScanItems && kAggPositions == 2u * kAggCutWindow,
              "the warps of k_count_scan find the cuts");
// The cuts (one more than blocks, found with the chain counts) and the internal
// cells that span one (from k_aggregate), as (cell, depth << 26 | simulation,
// first position), at most one per cut and depth.  Every range-th cut is an outer
// cut: a list per `range` blocks between two of them, and one of the cells that span
// an outer cut, which a single block combines.  128 blocks a range, but 256 above
// 2^21 bodies or so, where that single block is the longer part: the aggregates of
// 2^22 bodies 380 -> 359 us, of 2^24 1,385 -> 1,334, of 2^18 44 -> 46, of 700,001 95
// -> 97.
static uint32_t agg_range(uint32_t blocks) { return blocks > 8192u ? 256u : 128u; }
struct AggPlan {
    uint32_t* cuts;
    uint32_t* inner_n;  // [range], zeroed with the chain counts
    uint32_t* outer_n;  // zeroed with the control block
    uint4* inner;       // [range][16 blocks of a range]
    uint4* outer;       // [16 ranges]
    struct SpanCell* outer_cells;  // [16 ranges], with their links
    uint32_t blocks, range, ranges;
};

constexpr unsigned long long kScanAgg = 1ull << 62;
constexpr unsigned long long kScanInc = 2ull << 62;
constexpr unsigned long long kScanMask = (1ull << 62) - 1ull;

__global__ void __launch_bounds__(kScanThreads) k_count_scan(
    const SimDesc* __restrict__ sims, const uint32_t* __restrict__ chunk_sim, uint32_t npos,
    const uint32_t* __restrict__ codes, uint32_t* __restrict__ base, const AggPlan plan,
    uint32_t* tile_counter, unsigned long long* flags, uint32_t* err) {
    wait_for_predecessor();
    __shared__ uint32_t s_tile;
    __shared__ uint32_t s_scan[8];
    __shared__ unsigned long long s_excl;
    if (threadIdx.x == 0) s_tile = atomicAdd(tile_counter, 1u);
    __syncthreads();
    const uint32_t t = s_tile;
    const uint32_t p0 = t * kScanTile + threadIdx.x * kScanItems;
    uint32_t cnt[kScanItems];
    uint32_t sum = 0, cut = kNone;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const uint32_t p = p0 + k;
        uint32_t c = 0;
        if (p < npos) {
            const uint32_t s = chunk_sim[p >> 5];
            uint32_t dmin = 0;
            if (s != kNone) {
                const SimDesc& sd = sims[s];
                const uint32_t i = p - sd.off;
                if (i < sd.n)
                    c = chain_count(codes + sd.off, i, sd.n, sd.bucket, sd.max_depth, &dmin);
            }
            cut = min(cut, dmin << 16 | (p % kAggPositions));
        }
        cnt[k] = c;
        sum += c;
    }
    // a warp's positions are one half of a block's: a cut window, or not
    cut = __reduce_min_sync(kFull, cut);
    if (lane_id() == 0 && p0 % kAggPositions == 0u && p0 < npos)
        plan.cuts[p0 / kAggPositions] = p0 + (cut & 0xffffu);
    if (threadIdx.x == 0) {
        if (t == 0) plan.cuts[plan.blocks] = npos;
        if (t < plan.ranges) plan.inner_n[t] = 0;  // (a range spans many tiles)
    }
    uint32_t tile_total;
    const uint32_t texcl = block_exclusive_scan_256(sum, &tile_total, s_scan);
    if (threadIdx.x < 32u) {
        // decoupled look-back by one warp: lane j reads tile tp - j, so a
        // round covers 32 predecessors; a round counts once every tile up to
        // the nearest inclusive prefix has published (tiles before 0 read as
        // inclusive 0), otherwise it polls again (bounded)
        const uint32_t lane = threadIdx.x;
        unsigned long long excl = 0;
        if (t == 0) {
            if (lane == 0) atomicExch(&flags[0], kScanInc | (unsigned long long)tile_total);
        } else {
            if (lane == 0) atomicExch(&flags[t], kScanAgg | (unsigned long long)tile_total);
            long long tp = (long long)t - 1;
            const long long c0 = clock64();
            while (true) {
                const long long idx = tp - (long long)lane;
                const unsigned long long f = idx >= 0 ? ld_volatile64(&flags[idx]) : kScanInc;
                const unsigned long long st = f & ~kScanMask;
                const uint32_t inc = __ballot_sync(kFull, st == kScanInc);
                const uint32_t pub = __ballot_sync(kFull, st != 0ull);
                const uint32_t upto = inc ? (inc & (0u - inc)) * 2u - 1u : 0xffffffffu;
                if ((pub & upto) == upto) {
                    unsigned long long v = ((upto >> lane) & 1u) ? (f & kScanMask) : 0ull;
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
                    excl += v;
                    if (inc) break;
                    tp -= 32;
                } else if (__any_sync(kFull, clock64() - c0 > kSpinCycles)) {
                    if (lane == 0) set_err(err, kErrLookbackTimeout);
                    break;  // the whole warp: the vote is uniform
                }
            }
            if (lane == 0) atomicExch(&flags[t], kScanInc | (excl + tile_total));
        }
        if (lane == 0) s_excl = excl;
    }
    __syncthreads();
    uint32_t run = (uint32_t)s_excl + texcl;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const uint32_t p = p0 + k;
        if (p <= npos) base[p] = run;
        run += cnt[k];
    }
}

// ========================================================= small sort =====

// A simulation of at most kSmallSort bodies in one block or one cluster of up to
// 16: the step's integration (mode as k_integrate) and bounds, Morton codes, the
// four stable 8-bit passes in shared memory (a cluster's blocks write one
// another's), the gather into Morton order and, where the batch is that one
// simulation (SCAN), the chain counts and their scan.  Separate
// launches cost 10 us for the codes, 7 to 10 a pass and 10 for the scan however
// few keys they have: a launch, a chain of loads, a look-back, global stores.  A
// warp ranks its positions in order as k_radix_pass does (the lanes that share a
// digit by one ballot per digit bit); one block scan over (digit, blocks, warps)
// turns the counts into places, so the permutation is the same stable one.  In a
// cluster a block gets every block's digit counts before the scan, and an item
// goes straight to its place in whichever block has it: two barriers a pass, the
// first also the proof that every block has its items in registers.
// Bound by the barriers' latency (a pass of 16 blocks of 1,024 keys takes 10,000
// cycles: ranking 1,500, counts 2,000, the barriers 2,500 and 2,000, places 1,500)
// and, at 4,096 keys a block, by the 8-byte remote stores (5,000 of 19,000).  512
// threads have fewer counts to scan and fewer warps to wait for than 1,024, and
// shorter chains than 256: 92.6, 93.6 and 92.9 us a step at 16,384 bodies, 145, 146
// and 156 at 65,536.  Steps against separate launches: 4,096 bodies 121 -> 80 us (one
// block of 1,024 threads: 88), 8,192 112 -> 84, 16,384 117 -> 91, 32,768 128 -> 109,
// 65,536 154 -> 145.  With the integration and the bounds here too, and so no
// memset and no second reading of the positions, a rebuild takes 8 us less, a step
// 1,024 bodies 58 -> 56, 16,384 93 -> 92, 65,536 147 -> 148, 64 simulations of 16,384
// in a batch 705 -> 669.
constexpr int kSmallThreads = 512;
constexpr uint32_t kSmallBlocks = 16;  // most blocks of a cluster
static_assert(kSmallSort == kSmallBlocks * 4096u && kSmallSort <= 65536u,
              "body indices are kept in 16 bits");

template <int LOG>
struct SmallSort {
    uint64_t item[1 << LOG];  // body index << 32 | code
    // digit counts by warp, then first places (rows padded: the scan's
    // threads of a digit read rows 8 apart, in different banks)
    uint16_t place[kSmallThreads / 32][258];
    uint32_t digits[kSmallBlocks][264];  // the blocks' digit counts (padded likewise)
    float4 block_bounds[kSmallBlocks];   // the blocks' (min x, min y, max x, max y)
    float4 bounds[kSmallThreads / 32];   // the warps'
    uint32_t cells[kSmallBlocks];        // the blocks' chain counts
    uint32_t warp_sum[32];
    uint32_t cut[(1 << LOG) / kAggPositions];  // least dmin << 16 | position of the cut windows
};

// The cluster's barrier in its two halves (a block's exited threads count as
// arrived), and the address of a shared variable in another of its blocks.
__device__ __forceinline__ void cluster_arrive() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t peer_address(const void* shared, uint32_t block) {
    uint32_t at;
    asm("mapa.shared::cluster.u32 %0, %1, %2;"
        : "=r"(at)
        : "r"((uint32_t)__cvta_generic_to_shared(shared)), "r"(block));
    return at;
}

// The sorted codes, of which block b holds [b << LOG, (b + 1) << LOG).
template <int LOG>
struct ClusterCodes {
    const uint64_t* item;
    uint32_t block;
    __device__ __forceinline__ uint32_t operator[](uint32_t i) const {
        const uint64_t* at = item + (i & ((1u << LOG) - 1u));
        if (i >> LOG == block) return (uint32_t)*at;
        uint32_t v;
        asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(peer_address(at, i >> LOG)));
        return v;
    }
};

// Exclusive scan of one value per thread over a block of WARPS warps.
template <int WARPS>
__device__ __forceinline__ uint32_t small_scan(uint32_t v, uint32_t* warp_sum, uint32_t* total) {
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31u) warp_sum[warp] = x;
    __syncthreads();
    uint32_t w = lane < (uint32_t)WARPS ? warp_sum[lane] : 0u;  // every warp scans the warps' sums
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, w, o);
        if (lane >= (uint32_t)o) w += y;
    }
    *total = __shfl_sync(kFull, w, 31);
    const uint32_t before = __shfl_sync(kFull, w, (warp + 31u) & 31u);
    return x - v + (warp ? before : 0u);
}

template <int LOG, bool SCAN, bool CLUSTER, bool TIMED>
__global__ void __launch_bounds__(kSmallThreads) k_sort_small(
    const SimDesc* __restrict__ sims, int mode, uint32_t npos, uint32_t* __restrict__ keys,
    float4* __restrict__ sbody, uint32_t* __restrict__ base, const AggPlan plan, SimOut* simout,
    uint32_t* __restrict__ stage_cycles) {
    wait_for_predecessor();
    // TIMED: the stages in cycles of one thread: bounds, codes, sort with its
    // gather, chain counts with their scan.  A form of its own, for rebuilds whose
    // caller asks for times: the marks, and the gather done before the chain counts
    // start, cost a step 0.2 to 0.8 us (16,384 bodies 91.7 -> 92.2).
    uint32_t mark = TIMED ? (uint32_t)clock() : 0u;
    auto stage_done = [&](int stage) {
        if (TIMED && blockIdx.x == 0 && threadIdx.x == 0) {
            const uint32_t now = (uint32_t)clock();
            stage_cycles[stage] = now - mark;
            mark = now;
        }
    };
    extern __shared__ float4 small_shared[];
    SmallSort<LOG>& s = *reinterpret_cast<SmallSort<LOG>*>(small_shared);
    constexpr int ITEMS = (1 << LOG) / kSmallThreads;
    constexpr int kWarps = kSmallThreads / 32;
    constexpr int kParts = kSmallThreads / 256;  // threads of a digit, each with 8 warps' counts
    const uint32_t t = threadIdx.x, lane = lane_id(), warp = t >> 5;
    const uint32_t lanes_below = (1u << lane) - 1u;
    uint32_t block = 0, cluster = 1;
    if constexpr (CLUSTER) {
        asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(block));
        asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(cluster));
    }
    const uint32_t sim = blockIdx.x / cluster;
    const SimDesc& sd = sims[sim];
    const uint32_t first = block << LOG;
    if (CLUSTER && first >= sd.n) return;  // before any barrier
    const uint32_t blocks = (sd.n - 1u >> LOG) + 1u;
    const uint32_t n = min(sd.n - first, 1u << LOG);  // the block's positions
    if (CLUSTER) cluster_arrive();
    const uint32_t i0 = warp * (ITEMS * 32u) + lane;  // this thread's positions: i0 + 32 r
    if (SCAN && t < (1u << LOG) / kAggPositions) s.cut[t] = kNone;
    // the bodies moved (as k_integrate) and bounded, kBatch loads at a time
    constexpr int kBatch = ITEMS < 4 ? ITEMS : 4;
    float2 xy[ITEMS];
    float mnx = INFINITY, mny = INFINITY, mxx = -INFINITY, mxy = -INFINITY;
#pragma unroll
    for (int r0 = 0; r0 < ITEMS; r0 += kBatch) {
        float4 pm[kBatch], v[kBatch], acc[kBatch];
#pragma unroll
        for (int r = 0; r < kBatch; ++r) {
            const uint32_t i = i0 + 32u * (r0 + r);
            if (i >= n) continue;
            const float4* st = reinterpret_cast<const float4*>(sd.state + first + i);
            pm[r] = st[0];
            if (mode != 0) {
                v[r] = st[1];
                acc[r] = sd.accel[first + i];
            }
        }
#pragma unroll
        for (int r = 0; r < kBatch; ++r) {
            const uint32_t i = i0 + 32u * (r0 + r);
            if (i >= n) continue;
            if (mode != 0) {
                integrate(mode, sd.dt, pm[r], v[r], acc[r]);
                float4* st = reinterpret_cast<float4*>(sd.state + first + i);
                st[0] = pm[r];
                st[1] = v[r];
            }
            xy[r0 + r] = make_float2(pm[r].x, pm[r].y);
            mnx = fminf(mnx, pm[r].x);
            mny = fminf(mny, pm[r].y);
            mxx = fmaxf(mxx, pm[r].x);
            mxy = fmaxf(mxy, pm[r].y);
        }
    }
    auto reduce = [&]() {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            mnx = fminf(mnx, __shfl_xor_sync(kFull, mnx, o));
            mny = fminf(mny, __shfl_xor_sync(kFull, mny, o));
            mxx = fmaxf(mxx, __shfl_xor_sync(kFull, mxx, o));
            mxy = fmaxf(mxy, __shfl_xor_sync(kFull, mxy, o));
        }
    };
    auto gather = [&](const float4* bounds, uint32_t count) {  // each lane one, then all
        const float4 b = lane < count ? bounds[lane]
                                      : make_float4(INFINITY, INFINITY, -INFINITY, -INFINITY);
        mnx = b.x, mny = b.y, mxx = b.z, mxy = b.w;
        reduce();
    };
    reduce();
    if (lane == 0) s.bounds[warp] = make_float4(mnx, mny, mxx, mxy);
    __syncthreads();
    gather(s.bounds, kWarps);
    if constexpr (CLUSTER) {
        cluster_wait();  // every block runs: its shared memory may be written
        if (t < blocks)
            asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(
                             peer_address(&s.block_bounds[block], t)),
                         "f"(mnx), "f"(mny), "f"(mxx), "f"(mxy)
                         : "memory");
        cluster_arrive();
        cluster_wait();
        gather(s.block_bounds, blocks);
    }
    const RootBounds rb = root_bounds(mnx, mny, mxx, mxy);
    stage_done(0);
    if (t == 0 && block == 0) {
        simout[sim].cx = rb.cx;
        simout[sim].cy = rb.cy;
        simout[sim].half = rb.half;
        simout[sim].crit0 = crit_of(rb.half, sd.theta);
    }
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const uint32_t i = i0 + 32u * r;
        if (i < n)
            s.item[i] = (uint64_t)(first + i) << 32 |
                        morton2(quantize_axis((double)xy[r].x, rb.cx, rb.half),
                                quantize_axis((double)xy[r].y, rb.cy, rb.half));
    }
    stage_done(1);
    // a warp reads back only its own positions until the places are known
#pragma unroll 1
    for (uint32_t shift = 0; shift < 32u; shift += 8u) {
        uint32_t* row = reinterpret_cast<uint32_t*>(s.place[warp]);
        for (uint32_t k = lane; k < 129u; k += 32u) row[k] = 0u;
        __syncwarp();
        uint32_t key[ITEMS], val_rank[ITEMS];
#pragma unroll
        for (int r = 0; r < ITEMS; ++r) {
            const uint32_t i = i0 + 32u * r;
            const bool valid = i < n;
            const uint64_t item = valid ? s.item[i] : 0u;
            key[r] = (uint32_t)item;
            const uint32_t d = (key[r] >> shift) & 255u;
            uint32_t peers = __ballot_sync(kFull, valid);
#pragma unroll
            for (int bit = 0; bit < 8; ++bit) {
                const uint32_t m = __ballot_sync(kFull, (d >> bit) & 1u);
                peers &= ((d >> bit) & 1u) ? m : ~m;
            }
            const uint32_t leader = __ffs(peers) - 1u;
            uint32_t b = 0;
            if (valid && lane == leader) {
                b = s.place[warp][d];
                s.place[warp][d] = (uint16_t)(b + __popc(peers));
            }
            b = __shfl_sync(kFull, b, leader & 31u);
            val_rank[r] = (uint32_t)(item >> 32) | (b + __popc(peers & lanes_below)) << 16;
            __syncwarp();
        }
        __syncthreads();
        // thread kParts d + q: digit d of warps 8 q .. 8 q + 7
        const uint32_t d = t / kParts, q = t % kParts, w0 = q * 8u;
        uint32_t c[8], sum = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) c[w] = s.place[w0 + w][d];
#pragma unroll
        for (int w = 0; w < 8; ++w) sum += c[w];
        uint32_t total, at;
        if constexpr (CLUSTER) {
            // to the earlier threads of the digit in this block, those of the
            // blocks before it and the digits before it in all blocks
            uint32_t upto = sum;
#pragma unroll
            for (int o = 1; o < kParts; o <<= 1) {
                const uint32_t y = __shfl_up_sync(kFull, upto, o, kParts);
                if (q >= (uint32_t)o) upto += y;
            }
            const uint32_t mine = __shfl_sync(kFull, upto, kParts - 1, kParts);
            for (uint32_t to = q; to < blocks; to += kParts)
                asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(
                                 peer_address(&s.digits[block][d], to)),
                             "r"(mine)
                             : "memory");
            cluster_arrive();
            cluster_wait();
            uint32_t all = 0, before = 0;
            for (uint32_t b = q; b < blocks; b += kParts) {
                const uint32_t v = s.digits[b][d];
                all += v;
                if (b < block) before += v;
            }
#pragma unroll
            for (int o = 1; o < kParts; o <<= 1) {
                all += __shfl_xor_sync(kFull, all, o);
                before += __shfl_xor_sync(kFull, before, o);
            }
            at = small_scan<kWarps>(q == 0u ? all : 0u, s.warp_sum, &total);
            at = __shfl_sync(kFull, at, 0, kParts) + before + upto - sum;
        } else {
            at = small_scan<kWarps>(sum, s.warp_sum, &total);
        }
#pragma unroll
        for (int w = 0; w < 8; ++w) {
            s.place[w0 + w][d] = (uint16_t)at;
            at += c[w];
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < ITEMS; ++r) {
            if (i0 + 32u * r < n) {
                const uint32_t to = s.place[warp][(key[r] >> shift) & 255u] + (val_rank[r] >> 16);
                const uint64_t item = (uint64_t)(val_rank[r] & 0xffffu) << 32 | key[r];
                if constexpr (CLUSTER)
                    asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(peer_address(
                                     &s.item[to & ((1u << LOG) - 1u)], to >> LOG)),
                                 "l"(item)
                                 : "memory");
                else
                    s.item[to] = item;
            }
        }
        if constexpr (CLUSTER) {
            cluster_arrive();
            cluster_wait();
        } else {
            __syncthreads();
        }
    }
    const ClusterCodes<LOG> codes{s.item, block};
    float4 pm[ITEMS];  // the gather's loads are issued together
#pragma unroll
    for (int r = 0; r < ITEMS; ++r)
        if (i0 + 32u * r < n)
            pm[r] = __ldcg(reinterpret_cast<const float4*>(sd.state + (s.item[i0 + 32u * r] >> 32)));
    auto store = [&](int r, uint32_t i) {
        const uint64_t item = s.item[i];
        keys[sd.off + first + i] = (uint32_t)item;
        sbody[sd.off + first + i] =
            make_float4(pm[r].x, pm[r].y, pm[r].z, __uint_as_float((uint32_t)(item >> 32)));
    };
    if constexpr (TIMED) {
#pragma unroll
        for (int r = 0; r < ITEMS; ++r)
            if (i0 + 32u * r < n) store(r, i0 + 32u * r);
        stage_done(2);
    }
    uint32_t count[ITEMS], sum = 0;
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const uint32_t i = i0 + 32u * r;
        uint32_t cut = kNone;
        count[r] = 0;
        if (i < n) {
            if (!TIMED) store(r, i);
            if (SCAN) {
                uint32_t dmin;
                count[r] = chain_count(codes, first + i, sd.n, sd.bucket, sd.max_depth, &dmin);
                cut = dmin << 16 | (first + i);
            }
        }
        sum += count[r];
        if (SCAN && (i & ~31u) % kAggPositions < kAggCutWindow && (i & ~31u) < n) {
            cut = __reduce_min_sync(kFull, cut);
            if (lane == 0) atomicMin(&s.cut[i / kAggPositions], cut);
        }
    }
    if constexpr (SCAN) {  // cells per position, scanned in position order
        uint32_t total;
        sum = __reduce_add_sync(kFull, sum);  // the warp's
        uint32_t at = small_scan<kWarps>(lane ? 0u : sum, s.warp_sum, &total);
        at = __shfl_sync(kFull, at, 0);
        if constexpr (CLUSTER) {
            if (t < blocks)
                asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(
                                 peer_address(&s.cells[block], t)),
                             "r"(total)
                             : "memory");
            cluster_arrive();  // also the last access to a peer's memory
            cluster_wait();
            const uint32_t v = lane < blocks ? s.cells[lane] : 0u;
            at += __reduce_add_sync(kFull, lane < block ? v : 0u);
            total = __reduce_add_sync(kFull, v);
        }
#pragma unroll
        for (int r = 0; r < ITEMS; ++r) {
            uint32_t x = count[r];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(kFull, x, o);
                if (lane >= (uint32_t)o) x += y;
            }
            if (i0 + 32u * r < n) base[first + i0 + 32u * r] = at + x - count[r];
            at += __shfl_sync(kFull, x, 31);
        }
        if (block + 1u == blocks)
            for (uint32_t p = sd.n + t; p <= npos; p += kSmallThreads) base[p] = total;
        const uint32_t cut = first / kAggPositions + t;
        if (t < (1u << LOG) / kAggPositions && cut < plan.blocks)
            plan.cuts[cut] = s.cut[t] & 0xffffu;
        if (block == 0 && t == 0) plan.cuts[plan.blocks] = npos;
        if (block == 0 && t < plan.ranges) plan.inner_n[t] = 0;
        if (block == 0 && t == 0) *plan.outer_n = 0;
    }
    stage_done(3);
}

// =========================================================== aggregate ====

// Guard band of the f32 opening test.  The exact test (flat.rs:317-323) opens
// a cell unless width/dist < theta, i.e. approximates iff dist^2 > crit^2 with
// crit = width/theta.  The traversal computes d2 in f32 from the f32 centre of
// mass; with u = 2^-24 and C = |com_x| + |com_y| its error is at most
// 2u*C*d + 4u*d^2, and d <= (d^2 + crit^2)/(2 crit) turns that into a bound
// linear in d^2: |d2_f32 - d^2| <= d^2 * r + u*C*crit, r = u*C/crit + 4u.
// So d2_f32 > hi proves "approximate" and d2_f32 < lo proves "open" (with a
// 4x margin and 1e-4 relative slack); in between the traversal decides in f64.
// With r = u C/crit + 4 u the slack 4 r + 1e-4 on crit^2 and 4 u C crit beside
// it make crit^2 (16 u + 1e-4) + 8 u C crit on either side of crit^2; here in
// f32 with every rounding away from crit^2, so the band only widens (checked in
// exact arithmetic: it contains the band of the same formula in f64 for 200,000
// critical distances of 1e-30 to 1e19 and centres of as many magnitudes).
struct Crit {
    float up, down;  // width/theta rounded up and down; +inf at theta = 0 and beyond f32
};
__device__ __forceinline__ Crit crit_f32(double crit) {
    const float up = __double2float_ru(crit);
    return Crit{up, up < INFINITY ? __double2float_rd(crit) : INFINITY};
}
__device__ __forceinline__ void mac_band(Crit root, uint32_t depth, float com_x, float com_y,
                                         float* lo, float* hi) {
    const float scale = __uint_as_float((127u - depth) << 23);  // 2^-depth
    const float up = __fmul_ru(root.up, scale), down = __fmul_rd(root.down, scale);
    const float up2 = __fmul_ru(up, up);
    const float wide = __fmul_ru(__fmul_ru(up, 4.76837159e-7f), __fadd_ru(fabsf(com_x), fabsf(com_y)));
    const float down2 = __fmul_rd(down, down);
    // theta = 0, or a root's width/theta beyond f32: every finite d2 opens.  (Past
    // f32's end up2 is +inf, but down2, rounded down, its largest number: a smaller
    // d2 opens.  One that overflows is decided in f64 in either case.)
    const bool always_open = !(down2 < INFINITY);
    *hi = always_open ? INFINITY : __fmaf_ru(up2, 1.000101f, wide);
    *lo = always_open ? INFINITY : __fmaf_rd(down2, 0.999899f, -wide);
}

// hi with the depth in its low 5 bits, rounded away from zero to make room:
// a larger positive bound (or a more negative -1) only widens the band, and
// +inf becomes a NaN, for which "d2 > hi" stays false.
__device__ __forceinline__ float pack_depth(float hi, uint32_t depth) {
    return __uint_as_float(((__float_as_uint(hi) + 32u) & ~31u) | depth);
}

// Cell k's record for its slot of the parent's node group: internal cells get
// (hi|depth, lo); a leaf (count >= 1 bodies) is always summed directly: one
// body -> hi = -1 (it passes as a point mass at its own position, which is its
// f32 centre of mass exactly); several bodies -> hi = +inf (no point-mass
// term), summed body by body.  The slot's u = (lo | body count, start, body
// count, k or kNone for a leaf).  crit: the root's width/theta (halved at each
// depth).
__device__ __forceinline__ CellRec slot_record(uint32_t k, float fx, float fy, float gm,
                                               uint32_t depth, uint32_t start, uint32_t count,
                                               bool leaf, Crit crit) {
    float lo, hi;
    mac_band(crit, depth, fx, fy, &lo, &hi);
    if (leaf) hi = count == 1u ? -1.0f : INFINITY;
    const uint32_t ux = leaf ? count : __float_as_uint(lo);
    CellRec rec;
    rec.f = make_float4(fx, fy, gm, pack_depth(hi, depth));
    rec.u = make_uint4(ux, start, count, leaf ? kNone : k);
    return rec;
}

struct AggArgs {
    const SimDesc* sims;
    const SimOut* simout;
    const uint32_t* chunk_sim;
    const float4* sbody;
    const uint32_t* codes;
    uint32_t capacity;
    const uint32_t* base;
    uint4* cell_u;
    double4* cell_d;
    CellRec* groups;
    uint32_t nsims;
};

// The simulation a chunk of 32 positions belongs to, as the aggregates need it.
struct AggSim {
    Crit crit;            // root width / theta
    uint32_t off, end;    // its positions (end = 0: an unused chunk)
    uint32_t root_group;  // capacity + sim
    float g;
};

// Mass and centre of mass of a cell from its weighted sums, as
// nbody/src/flat.rs:193-212, in f64.
struct CellSum {
    double mass = 0.0, wx = 0.0, wy = 0.0;  // then wx, wy become the centre of mass
    __device__ __forceinline__ void add(double m, double x, double y) {
        mass = __dadd_rn(mass, m);
        wx = __dadd_rn(wx, __dmul_rn(m, x));
        wy = __dadd_rn(wy, __dmul_rn(m, y));
    }
    __device__ __forceinline__ void finish() {
        wx = __ddiv_rn(wx, mass);
        wy = __ddiv_rn(wy, mass);
    }
};

// Writes a finished cell's f64 record; returns its centre of mass in f32.
__device__ __forceinline__ float2 store_cell(double4* cell_d, uint32_t k, const CellSum& c) {
    const float hx = (float)c.wx, hy = (float)c.wy;
    // the f32 residuals com - (float)com ride in the record's spare word: the
    // compensated traversal adds them back to its differences
    const float lo_x = (float)(c.wx - (double)hx), lo_y = (float)(c.wy - (double)hy);
    const unsigned long long lo_bits =
        ((unsigned long long)__float_as_uint(lo_y) << 32) | __float_as_uint(lo_x);
    cell_d[k] = make_double4(c.wx, c.wy, c.mass, __longlong_as_double((long long)lo_bits));
    return make_float2(hx, hy);
}

// Bottom-up f64 aggregates.  The structure below a run of positions needs no
// links: position p starts a group at every depth >= dmin(p) (one more than
// the levels it shares with p - 1), its cells are numbered base[p] + d -
// dmin(p), and a group ends at the next position whose dmin is at most its
// depth.  A block owns the cells that start between two cuts.  It computes
// every leaf, then the internal cells that end before the next cut, depth by
// depth, deepest first, with a block barrier between depths.  The sum and end
// of the last cell done at each position stay in shared memory, so a cell
// hops over its children there (the first at its own start, the next at each
// child's end), and it writes its whole node group, a 128-byte line; nothing
// is loaded from global memory after the block's codes, bases and bodies.  The
// cells that span a cut (few, and shallow: the cuts lie at the coarsest group
// starts near every kAggPositions) are listed for k_aggregate_inner.  A leaf sums
// its bodies in Morton order, an internal cell its children in quadrant order
// 0..3 (nbody/src/flat.rs:179-215): the f64 mass and centre of mass equal the
// reference's bit for bit.
//
// What bounds it: the chain of depths (about 700 cycles each: a few dependent
// shared loads, four sums, two divisions, a barrier), at 8 blocks of 4 warps
// per SM.  Links and values read from global memory per cell, with a climb
// through an acquire-release counter wherever a parent crossed a block, took
// 156 us at 2^20 bodies (458 at 2^22, 61 at 2^14, 45 at 2^10); this and
// the spanning cells' passes took 110 (331, 28, 20), and with the links as well,
// for which a cells kernel took another 64 (239), 122 (361, 32, 22).  Before the
// links, 256 threads: 130 us at 2^20, 64: 140; four lanes per cell: 168; cut windows
// of 64 and 256 positions: 112, 118.
#ifndef GBH_AGG_THREADS
#define GBH_AGG_THREADS 128
#endif
#ifndef GBH_AGG_MIN_BLOCKS
#define GBH_AGG_MIN_BLOCKS 8
#endif
constexpr uint32_t kAggThreads = GBH_AGG_THREADS;
constexpr uint32_t kAggItems = kAggPositions + kAggCutWindow;  // positions of a block, at most
constexpr uint32_t kAggGroups = (kAggItems + 31u) / 32u;

__device__ __forceinline__ AggSim agg_sim(const AggArgs& a, uint32_t sim) {
    AggSim si{};
    if (sim != kNone) {
        const SimDesc& sd = a.sims[sim];
        si.crit = crit_f32(a.simout[sim].crit0);
        si.off = sd.off;
        si.end = sd.off + sd.n;
        si.root_group = a.capacity + sim;
        si.g = sd.g_f;
    }
    return si;
}

// One child of a cell, or none, as its slot of the cell's node group: an
// absent child takes the lowest quadrant left in `missing`.
__device__ __forceinline__ void store_child(const AggArgs& a, uint32_t parent, bool have,
                                            uint32_t quadrant, uint32_t* missing, uint32_t k,
                                            float x, float y, float gm, uint32_t depth,
                                            uint32_t start, uint32_t end, bool leaf, Crit crit) {
    CellRec rec = slot_record(k, x, y, gm, depth, start, end - start, leaf, crit);
    if (!have) {
        rec.f = make_float4(0.f, 0.f, 0.f, 0.f);
        rec.u = make_uint4(0u, 0u, 0u, kNone);
        quadrant = __ffs(*missing) - 1u;
        *missing &= *missing - 1u;
    }
    CellRec* group = a.groups + 4ull * parent;
    group[quadrant].f = rec.f;
    group[quadrant].u = rec.u;
}

// A root: slot 0 of its simulation's root group, the other slots empty.
__device__ __forceinline__ void store_root(const AggArgs& a, uint32_t root_group, uint32_t k,
                                           float x, float y, float gm, uint32_t start,
                                           uint32_t end, bool leaf, Crit crit) {
    CellRec* group = a.groups + 4ull * root_group;
    group[0] = slot_record(k, x, y, gm, 0u, start, end - start, leaf, crit);
#pragma unroll
    for (int q = 1; q < 4; ++q) group[q].u = make_uint4(0u, 0u, 0u, kNone);
}

// End of the depth-d group that starts before position lo and goes on to it, by
// code prefix (d levels of `code`), at most hi.
__device__ __forceinline__ uint32_t group_end(const uint32_t* codes, uint32_t lo, uint32_t hi,
                                              uint32_t code, uint32_t d) {
    if (d == 0u) return hi;
    const uint32_t sh = 32u - 2u * d;
    const unsigned long long next = ((unsigned long long)(code >> sh) + 1ull) << sh;
    if (next > 0xffffffffull) return hi;
    const uint32_t x[1] = {(uint32_t)next};
    uint32_t out[1];
    kary_lower_bound<1>(codes, lo, hi, x, out);
    return out[0];
}

struct AggShared {
    // the last finished cell that starts at position i: centre of mass x, y and
    // mass (f64), then its end | dmin of that end << 16 (positions of the block)
    double x[kAggItems], y[kAggItems], m[kAggItems];
    float fx[kAggItems], fy[kAggItems], gm[kAggItems];  // in f32, with G*mass
    uint32_t link[kAggItems];
    uint32_t code[kAggItems];
    uint32_t base[kAggItems + 1];
    // dmin | depth of the chain's leaf << 8 | first depth whose group ends
    // inside the block << 16
    uint32_t info[kAggItems + 1];
    AggSim sim[kAggGroups + 1];  // by chunk of 32 positions
    // local internal cells by depth, as positions: those of one depth hold
    // disjoint ranges of at least two positions
    uint16_t level[kMortonDepth][kAggItems / 2u];
    uint16_t count[kAggGroups][kMortonDepth], total[kMortonDepth];
    uint32_t depths;  // depths that have some
};

__global__ void __launch_bounds__(kAggThreads, GBH_AGG_MIN_BLOCKS)
    k_aggregate(const AggArgs a, const AggPlan plan, uint32_t* err) {
    wait_for_predecessor();
    __shared__ AggShared s;
    const uint32_t t = threadIdx.x, lane = lane_id(), warp = t >> 5;
    const bool stop = gave_up(err);  // (no block of this kernel sets that bit)
    const uint32_t R0 = plan.cuts[blockIdx.x], R1 = plan.cuts[blockIdx.x + 1u];
    const uint32_t npos = plan.cuts[plan.blocks];
    const uint32_t n = R1 - R0;
    if (n - 1u >= kAggItems) {  // cannot be: the cuts lie in windows
        if (t == 0) set_err(err, kErrCapacity);
        return;
    }
    const uint32_t chunk0 = R0 >> 5;
    for (uint32_t j = t; j < n; j += kAggThreads) {
        s.code[j] = a.codes[R0 + j];
        s.base[j] = a.base[R0 + j];
    }
    if (t <= (R1 - 1u) / 32u - chunk0) s.sim[t] = agg_sim(a, a.chunk_sim[chunk0 + t]);
    const uint32_t before = R0 > 0u ? a.codes[R0 - 1u] : 0u;
    const uint32_t after = R1 < npos ? a.codes[R1] : 0u;
    const uint32_t range = blockIdx.x / plan.range;
    const uint32_t R2 = plan.cuts[min((range + 1u) * plan.range, plan.blocks)];  // the outer cut
    const uint32_t beyond = R2 < npos ? a.codes[R2] : 0u;
    if (t == 0) {
        s.depths = 0;
        s.info[n] = 0;
        s.base[n] = a.base[R1];
    }
    __syncthreads();
    if (stop) {
        // no cells and no lists (the list passes find them empty), and root groups
        // without a root: the traversal then has nothing to read
        if (blockIdx.x == 0)
            for (uint32_t k = t; k < 4u * a.nsims; k += kAggThreads)
                a.groups[4ull * a.capacity + k].u = make_uint4(0u, 0u, 0u, kNone);
        return;
    }
    if (s.base[n] > a.capacity) {  // cannot be: the capacity bounds every tree
        if (t == 0) set_err(err, kErrCapacity);
        return;
    }
    const uint32_t groups = (n + 31u) / 32u;
    auto local = [](uint32_t info, uint32_t d) {
        return d >= ((info >> 16) & 0xffu) && d < ((info >> 8) & 0xffu);
    };
    auto sim_of = [&](uint32_t j) -> const AggSim& { return s.sim[((R0 + j) >> 5) - chunk0]; };
    for (uint32_t g = warp; g < groups; g += kAggThreads / 32u) {
        const uint32_t j = g * 32u + lane, p = R0 + j;
        uint32_t depths = 0;
        if (j < n) {
            const AggSim& si = sim_of(j);
            const uint32_t code = s.code[j], cells = s.base[j + 1u] - s.base[j];
            // positions past the simulation's end head every depth: they end its groups
            uint32_t dmin = 0, deepest = 0;
            if (p < si.end && p != si.off)
                dmin = shared_levels(j ? s.code[j - 1u] : before, code) + 1u;
            if (cells) deepest = dmin + cells - 1u;
            const uint32_t dlo = si.end > R1 ? max(dmin, shared_levels(code, after) + 1u) : dmin;
            s.info[j] = dmin | deepest << 8 | dlo << 16;
            if (deepest > dlo) depths = ((1u << deepest) - 1u) & ~((1u << dlo) - 1u);
            for (uint32_t d = dmin; d < min(dlo, deepest); ++d) {  // the cells that span R1
                const uint4 rec = make_uint4(s.base[j] + d - dmin,
                                             d << 26 | (si.root_group - a.capacity), p, 0u);
                if (si.end > R2 && shared_levels(code, beyond) >= d)
                    plan.outer[atomicAdd(plan.outer_n, 1u)] = rec;
                else
                    plan.inner[(size_t)range * 16u * plan.range + atomicAdd(plan.inner_n + range, 1u)] =
                        rec;
            }
        }
        depths = __reduce_or_sync(kFull, depths);
        if (lane == 0 && depths) atomicOr(&s.depths, depths);
    }
    __syncthreads();
    for (uint32_t j = t; j < n; j += kAggThreads) {
        const uint32_t k = s.base[j + 1u] - 1u;
        if (s.base[j + 1u] == s.base[j]) continue;
        const uint32_t info = s.info[j], d = (info >> 8) & 0xffu;
        const AggSim& si = sim_of(j);
        const float4 body = a.sbody[R0 + j];
        CellSum sum;
        sum.add((double)body.z, (double)body.x, (double)body.y);
        uint32_t q = j + 1u;
        for (; (s.info[q] & 0xffu) > d; ++q) {  // s.info[n] = 0 ends the walk
            const float4 b = a.sbody[R0 + q];
            sum.add((double)b.z, (double)b.x, (double)b.y);
        }
        s.link[j] = q | (s.info[q] & 0xffu) << 16;
        uint32_t end = R0 + q;
        if (q == n && d < ((info >> 16) & 0xffu)) {  // the leaf goes on past the block
            end = group_end(a.codes, R1, si.end, s.code[j], d);
            for (uint32_t g = R0 + q; g < end; ++g) {
                const float4 b = a.sbody[g];
                sum.add((double)b.z, (double)b.x, (double)b.y);
            }
        }
        float2 com = make_float2(body.x + 0.f, body.y + 0.f);
        float mass = body.z;
        if (end == R0 + j + 1u) {
            // one body: m x of two f32 values is exact in f64, so (m x) / m is x
            // (+0.0 for -0.0, as the sum that starts at +0.0)
            sum.wx = (double)com.x;
            sum.wy = (double)com.y;
            a.cell_d[k] = make_double4(sum.wx, sum.wy, sum.mass, 0.0);
        } else {
            sum.finish();
            com = store_cell(a.cell_d, k, sum);
            mass = (float)sum.mass;
        }
        s.x[j] = sum.wx;
        s.y[j] = sum.wy;
        s.m[j] = sum.mass;
        s.fx[j] = com.x;
        s.fy[j] = com.y;
        s.gm[j] = __fmul_rn(si.g, mass);
        a.cell_u[k] = make_uint4(end, k + 1u, R0 + j, d);
        if (d == 0u)  // the simulation is one leaf
            store_root(a, si.root_group, k, com.x, com.y, s.gm[j], R0 + j, end, true, si.crit);
    }
    // the cells of each depth, in position order: counts by group of 32
    // positions, then every group's places
    const uint32_t depths = s.depths;
    for (uint32_t g = warp; g < groups; g += kAggThreads / 32u) {
        const uint32_t info = g * 32u + lane < n ? s.info[g * 32u + lane] : 0u;
        uint32_t count = 0;
        for (uint32_t m = depths; m; m &= m - 1u) {
            const uint32_t d = __ffs(m) - 1u;
            const uint32_t votes = __popc(__ballot_sync(kFull, local(info, d)));
            if (lane == d) count = votes;
        }
        if (lane < kMortonDepth) s.count[g][lane] = (uint16_t)count;
    }
    __syncthreads();
    for (uint32_t g = warp; g < groups; g += kAggThreads / 32u) {
        const uint32_t info = g * 32u + lane < n ? s.info[g * 32u + lane] : 0u;
        uint32_t place = 0;
        if (lane < kMortonDepth) {
            for (uint32_t q = 0; q < g; ++q) place += s.count[q][lane];
            if (g + 1u == groups) s.total[lane] = (uint16_t)(place + s.count[g][lane]);
        }
        for (uint32_t m = depths; m; m &= m - 1u) {
            const uint32_t d = __ffs(m) - 1u;
            const uint32_t votes = __ballot_sync(kFull, local(info, d));
            const uint32_t at = __shfl_sync(kFull, place, d) + __popc(votes & ((1u << lane) - 1u));
            if ((votes >> lane) & 1u) s.level[d][at] = (uint16_t)(g * 32u + lane);
        }
    }
    __syncthreads();
    // The cells of one depth, a thread each.  No branch on the children: an
    // absent one stands in as the first and adds 0 (lanes taking turns at four
    // ways through the code cost more than the arithmetic).  The node group is
    // written after the depth's barrier, and the next depth's cells go to other
    // warps first, so the stores are off the way from depth to depth: children
    // but the first are final, and the first's values are kept (`first`).
    struct {
        uint32_t d = kNone, c0 = 0, c1 = 0, c2 = 0, c3 = 0, kids = 0, link0 = 0;
        float fx = 0.f, fy = 0.f, gm = 0.f;
    } first;
    auto store_group = [&]() {
        const uint32_t d = first.d;
        if (d == kNone) return;
        const uint32_t c[4] = {first.c0, first.c1, first.c2, first.c3};
        const uint32_t k = s.base[first.c0] + d - (s.info[first.c0] & 0xffu);
        const AggSim& sim = sim_of(first.c0);
        uint32_t quadrant[4], missing = 15u;
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q) {
            quadrant[q] = (s.code[c[q]] >> (30u - 2u * d)) & 3u;
            missing &= ~(1u << quadrant[q]);  // (an absent child repeats the first)
        }
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q) {
            const uint32_t kid = s.base[c[q]] + d + 1u - (s.info[c[q]] & 0xffu);
            const uint32_t link = q ? s.link[c[q]] : first.link0;
            store_child(a, k, q < first.kids, quadrant[q], &missing, kid,
                        q ? s.fx[c[q]] : first.fx, q ? s.fy[c[q]] : first.fy,
                        q ? s.gm[c[q]] : first.gm, d + 1u, R0 + c[q], R0 + (link & 0xffffu),
                        kid + 1u == s.base[c[q] + 1u], sim.crit);
        }
        first.d = kNone;
    };
    uint32_t turn = 0;
    for (uint32_t todo = depths; todo != 0u;) {
        const uint32_t d = 31u - __clz(todo);
        todo &= ~(1u << d);
        const uint32_t cells = s.total[d];
        for (uint32_t i = (t + turn) % kAggThreads; i < cells; i += kAggThreads) {
            store_group();
            const uint32_t c0 = s.level[d][i];
            const uint32_t k = s.base[c0] + d - (s.info[c0] & 0xffu);
            const uint32_t link0 = s.link[c0];
            const bool two = (link0 >> 16) > d;
            const uint32_t c1 = two ? link0 & 0xffffu : c0;
            const uint32_t link1 = s.link[c1];
            const bool three = two && (link1 >> 16) > d;
            const uint32_t c2 = three ? link1 & 0xffffu : c0;
            const uint32_t link2 = s.link[c2];
            const bool four = three && (link2 >> 16) > d;
            const uint32_t c3 = four ? link2 & 0xffffu : c0;
            const uint32_t link3 = s.link[c3];
            const uint32_t c[4] = {c0, c1, c2, c3};
            const bool have[4] = {true, two, three, four};
            CellSum sum;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                // (adding 0.0 leaves a sum: it starts at +0.0 and is never -0.0)
                const double m = s.m[c[q]];
                sum.mass = __dadd_rn(sum.mass, have[q] ? m : 0.0);
                sum.wx = __dadd_rn(sum.wx, have[q] ? __dmul_rn(m, s.x[c[q]]) : 0.0);
                sum.wy = __dadd_rn(sum.wy, have[q] ? __dmul_rn(m, s.y[c[q]]) : 0.0);
            }
            first.d = d;
            first.c0 = c0;
            first.c1 = c1;
            first.c2 = c2;
            first.c3 = c3;
            first.kids = 1u + two + three + four;
            first.link0 = link0;
            first.fx = s.fx[c0];
            first.fy = s.fy[c0];
            first.gm = s.gm[c0];
            sum.finish();
            s.x[c0] = sum.wx;
            s.y[c0] = sum.wy;
            s.m[c0] = sum.mass;
            const uint32_t link = four ? link3 : three ? link2 : two ? link1 : link0;
            s.link[c0] = link;
            const AggSim& sim = sim_of(c0);
            const float2 com = store_cell(a.cell_d, k, sum);
            const uint32_t end = link & 0xffffu;
            a.cell_u[k] = make_uint4(R0 + end, s.base[end], R0 + c0, d);
            const float gm = __fmul_rn(sim.g, (float)sum.mass);
            s.fx[c0] = com.x;
            s.fy[c0] = com.y;
            s.gm[c0] = gm;
            if (d == 0u)
                store_root(a, sim.root_group, k, com.x, com.y, gm, R0 + c0, R0 + end, false, sim.crit);
        }
        __syncthreads();
        store_group();
        turn += kAggThreads / 2u;
    }
}

// One cell that spans a cut: its links by searches over the codes, its sums from
// its children's f64 records.
struct SpanCell {
    uint32_t k, depth, start, end, c[4];
    uint32_t kid_end[4], kid_start[4];
    bool kid_leaf[4];
    AggSim sim;

    // limit: a position its end does not pass
    __device__ __forceinline__ void load(const AggArgs& a, uint4 rec, uint32_t limit) {
        k = rec.x;
        depth = rec.y >> 26;
        start = rec.z;
        const SimDesc& sd = a.sims[rec.y & 0x3ffffffu];
        sim = agg_sim(a, rec.y & 0x3ffffffu);
        const uint32_t code = a.codes[start];
        end = group_end(a.codes, start + 1u, min(sim.end, limit), code, depth);
        const uint32_t sh = 30u - 2u * depth;
        const uint32_t prefix = depth == 0u ? 0u : (code >> (sh + 2u)) << 2;
        const uint32_t x[3] = {(prefix | 1u) << sh, (prefix | 2u) << sh, (prefix | 3u) << sh};
        uint32_t bound[3];
        kary_lower_bound<3>(a.codes, start, end, x, bound);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            kid_start[q] = q ? bound[q - 1] : start;
            kid_end[q] = q < 3 ? bound[q] : end;
            // the first child follows its parent, the others head their positions' chains
            c[q] = kid_start[q] == kid_end[q] ? kNone
                   : kid_start[q] == start    ? k + 1u
                                              : a.base[kid_start[q]];
            kid_leaf[q] = kid_end[q] - kid_start[q] <= sd.bucket || depth + 1u >= sd.max_depth;
        }
        a.cell_u[k] = make_uint4(end, a.base[end], start, depth);
    }
    __device__ __forceinline__ void combine(const AggArgs& a) const {
        CellSum sum;
        double2 com[4];
        double m[4];
        uint32_t missing = 15u;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const double4* rec = a.cell_d + (c[q] == kNone ? k + 1u : c[q]);
            com[q] = __ldcg(reinterpret_cast<const double2*>(rec));
            m[q] = __ldcg(reinterpret_cast<const double*>(rec) + 2);
            if (c[q] != kNone) missing &= ~(1u << q);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (c[q] != kNone) sum.add(m[q], com[q].x, com[q].y);
        sum.finish();
        const float2 own = store_cell(a.cell_d, k, sum);
#pragma unroll
        for (int q = 0; q < 4; ++q)
            store_child(a, k, c[q] != kNone, (uint32_t)q, &missing, c[q], (float)com[q].x,
                        (float)com[q].y, __fmul_rn(sim.g, (float)m[q]), depth + 1u, kid_start[q],
                        kid_end[q], kid_leaf[q], sim.crit);
        if (depth == 0u)
            store_root(a, sim.root_group, k, own.x, own.y, __fmul_rn(sim.g, (float)sum.mass), start,
                       end, false, sim.crit);
    }
};

// The cells of a list that span cuts, depth by depth: each depth waits for the
// one below, and a barrier of one block is the cheapest wait.  A thread per cell,
// everything but the children's sums in hand before the first depth (the further
// cells of a list longer than the block are fetched in turn).
template <typename Fetch>
__device__ __forceinline__ void combine_spans(const AggArgs& a, uint32_t n, Fetch fetch) {
    __shared__ uint32_t s_depths;
    const uint32_t t = threadIdx.x;
    if (t == 0) s_depths = 0;
    __syncthreads();
    SpanCell cell;
    cell.depth = kNone;
    for (uint32_t i = t; i < n; i += blockDim.x) {
        SpanCell c;
        fetch(i, &c);
        atomicOr(&s_depths, 1u << c.depth);
        if (i == t) cell = c;
    }
    __syncthreads();
    for (uint32_t todo = s_depths; todo != 0u;) {
        const uint32_t d = 31u - __clz(todo);
        todo &= ~(1u << d);
        if (cell.depth == d) cell.combine(a);
        for (uint32_t i = t + blockDim.x; i < n; i += blockDim.x) {
            SpanCell more;
            fetch(i, &more);
            if (more.depth == d) more.combine(a);
        }
        __syncthreads();
    }
}

#ifndef GBH_SPAN_THREADS
#define GBH_SPAN_THREADS 512
#endif
constexpr uint32_t kSpanThreads = GBH_SPAN_THREADS;

// The lists of the inner cuts, a block each; the blocks after them find the
// links of the cells that span outer cuts meanwhile.
__global__ void __launch_bounds__(kSpanThreads) k_aggregate_inner(const AggArgs a,
                                                                  const AggPlan plan) {
    wait_for_predecessor();
    const uint32_t r = blockIdx.x;
    if (r >= plan.ranges) {
        const uint32_t n = min(*plan.outer_n, kMortonDepth * plan.ranges);
        const uint32_t i = (r - plan.ranges) * kSpanThreads + threadIdx.x;
        if (i < n) plan.outer_cells[i].load(a, plan.outer[i], kNone);
        return;
    }
    const uint4* list = plan.inner + (size_t)r * 16u * plan.range;
    const uint32_t n = min(plan.inner_n[r], 16u * plan.range);
    if (n == 0u) return;
    const uint32_t outer_cut = plan.cuts[min((r + 1u) * plan.range, plan.blocks)];
    combine_spans(a, n, [&](uint32_t i, SpanCell* c) { c->load(a, list[i], outer_cut); });
}

// Then the list of the outer cuts: in a single list with the inner ones, the
// cells of 2^20 bodies took 70 us instead of 11 and 14.
__global__ void __launch_bounds__(kSpanThreads) k_aggregate_outer(const AggArgs a,
                                                                  const AggPlan plan) {
    wait_for_predecessor();
    const uint32_t n = min(*plan.outer_n, kMortonDepth * plan.ranges);
    combine_spans(a, n, [&](uint32_t i, SpanCell* c) { *c = plan.outer_cells[i]; });
}

// Recomputes G*m and the MAC bands of one simulation from the f64 aggregates,
// for a force pass whose theta or G differs from the rebuild's: a thread per
// cell, its children's slots (child k + 1, then each at the one before's skip).
__global__ void k_refresh_mac(const SimDesc* __restrict__ sims, const SimOut* __restrict__ simout,
                              uint32_t sim, const uint32_t* __restrict__ base,
                              const uint32_t* __restrict__ codes, uint32_t capacity,
                              const double4* __restrict__ cell_d,
                              const uint4* __restrict__ cell_u, CellRec* groups) {
    const SimDesc& sd = sims[sim];
    const uint32_t cb = base[sd.off], ce = base[sd.off + sd.n];
    const uint32_t k = cb + blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= ce) return;
    const Crit crit = crit_f32(crit_of(simout[sim].half, sd.theta));
    auto store = [&](CellRec* slot, uint32_t c, const uint4& u) {
        const double4 v = cell_d[c];
        *slot = slot_record(c, (float)v.x, (float)v.y, __fmul_rn(sd.g_f, (float)v.z), u.w, u.z,
                            u.x - u.z, u.y == c + 1u, crit);
    };
    const uint4 u = cell_u[k];
    if (k == cb) store(groups + 4ull * (capacity + sim), k, u);
    for (uint32_t c = k + 1u; c < u.y;) {  // a leaf's skip is k + 1
        const uint4 cu = cell_u[c];
        store(groups + 4ull * k + ((codes[cu.z] >> (30u - 2u * u.w)) & 3u), c, cu);
        c = cu.y;
    }
}

// ============================================================ traverse ====

// Paired f32 arithmetic (sm_100 FADD2 / FFMA2 / FMUL2) for the compensated
// form: both axes of a term in one instruction, each axis rounded exactly as
// its scalar operation; a - b is fma(b, -1, a) (exact negation, one
// rounding).  The plain form keeps scalar operations (paired ones measured
// slower there: 0.667 against 0.592 ms at N = 2^20).
template <bool PAIRED>
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
    if (PAIRED) return __ffma2_rn(b, make_float2(-1.f, -1.f), a);
    return make_float2(a.x - b.x, a.y - b.y);
}

template <bool COMP>
struct Acc {
    float2 v = make_float2(0.f, 0.f);  // the sum (x, y)
    float2 c = make_float2(0.f, 0.f);  // compensated form: the two-sum error terms
    // adds the term d * scale: the plain form with one fused multiply-add per
    // axis, the compensated form with the rounded product and Knuth's two-sum
    // (s + e == v + t exactly)
    __device__ __forceinline__ void add_scaled(float2 d, float scale) {
        if (COMP) {
            const float2 t = __fmul2_rn(d, make_float2(scale, scale));
            const float2 s = __fadd2_rn(v, t);
            const float2 bb = sub2<true>(s, v);
            c = __fadd2_rn(c, __fadd2_rn(sub2<true>(v, sub2<true>(s, bb)), sub2<true>(t, bb)));
            v = s;
        } else {
            v.x += d.x * scale;
            v.y += d.y * scale;
        }
    }
    __device__ __forceinline__ float fx() const { return COMP ? v.x + c.x : v.x; }
    __device__ __forceinline__ float fy() const { return COMP ? v.y + c.y : v.y; }
};

// Lane-parallel traversal with interaction lists.  A warp owns 32
// consecutive Morton positions (its lanes).  Every lane keeps exactly its
// own opening decisions of nbody/src/flat.rs:270-346, but the walk itself is
// spread over the lanes: the warp pops up to 8 (node group, lane mask)
// entries from a per-warp stack in shared memory, and lane 4i+q examines
// slot q of popped entry i for all lanes of its mask at once, against the
// bounding box of the warp's bodies:
//   * the box's nearest point has d2 > hi: every lane of the mask
//     approximates the cell (a lane whose own body the cell holds opens it);
//   * the box's farthest corner has d2 < lo: every lane of the mask opens it;
//   * otherwise the cell is mixed and the warp decides it lane by lane, as
//     a single lane would (f64 test inside the guard band).
// d2 is fma(dx, dx, dy*dy) in f32 with round-to-nearest, monotone in |dx|
// and |dy|, and each lane's |dx|, |dy| lie between the box's nearest and
// farthest distances, so a box decision is every lane's own decision.
// Approximated cells and one-body leaves go to a per-warp interaction list
// (centre of mass, G*m, mask of the lanes that take the term), which all
// lanes sum with one branch-free masked term per entry; mixed cells add
// their term directly and leaves of several bodies are summed body by body,
// self excluded.  Only the order of a lane's terms differs from the
// reference's depth-first order.

// Exact f64 opening test of flat.rs:317-323 for a lane inside the guard
// band; true = approximate.
__device__ __noinline__ bool exact_mac(const double4* __restrict__ cell_d, uint32_t c, float tx,
                                       float ty, double root_half, uint32_t depth,
                                       double theta) {
    const double2 com = *reinterpret_cast<const double2*>(cell_d + c);
    const double ddx = __dsub_rn(com.x, (double)tx);
    const double ddy = __dsub_rn(com.y, (double)ty);
    const double dist = hypot(ddx, ddy);
    const double width = __dmul_rn(__dmul_rn(root_half, pow2_neg(depth)), 2.0);
    return dist > 0.0 && __ddiv_rn(width, dist) < theta;
}

// Squared distance as the traversal computes it everywhere (monotone in |dx|
// and |dy|; its rounding is covered by the guard band of mac_band).
__device__ __forceinline__ float dist2(float dx, float dy) {
    return __fmaf_rn(dx, dx, __fmul_rn(dy, dy));
}

// Lane mask of bits [a, b), 0 <= a <= b <= 32.
__device__ __forceinline__ uint32_t bit_range(uint32_t a, uint32_t b) {
    const uint32_t w = b - a;
    return w >= 32u ? 0xffffffffu : (((1u << w) - 1u) << a);
}

#ifndef GBH_TRAVERSE_WARPS
#define GBH_TRAVERSE_WARPS 8
#endif
#ifndef GBH_TRAVERSE_MIN_BLOCKS
#define GBH_TRAVERSE_MIN_BLOCKS 4  // 64 registers: 32 warps per SM
#endif
constexpr uint32_t kTravWarps = GBH_TRAVERSE_WARPS;
// Stack bound.  Each step pops the top <= 8 entries and pushes the opened
// children groups (<= 32) in the order of their parents' stack positions, so
// the stack stays sorted by depth with the deepest entries on top.  When
// entries of depth d are pushed, every earlier entry of depth d has already
// been popped (it sat above the depth d-1 parent), so at most 32 entries of
// one depth are held at once.  Groups belong to the 16 internal depths 0..15
// (Morton codes resolve 16 levels) or are a root group: 17 depths.
constexpr uint32_t kTravStack = 17u * 32u;
// Interaction list: flushed once it holds >= 32 entries; a step adds <= 32.
constexpr uint32_t kTravList = 64u;
static_assert(kTravList >= 64u, "the mixed cells of a step park in list[32, 64)");

// Reciprocal square root of a softened squared distance.  NORMAL: the squared
// softening is a normal number, so no such distance is subnormal, and the
// instruction without the subnormals' rescaling (about three more instructions
// of the ~15 of a term) gives the same bits.  The traversal is issue-bound: at
// 2^20 bodies 588 -> 541 us (theta 0.5), 2^22 compensated 3818 -> 3614, 700,001
// at theta 0.12 2704 -> 2469.  A template of the
// kernel, chosen on the host: both forms in one kernel spilled (609 us).
template <bool NORMAL>
__device__ __forceinline__ float rsqrt_r2(float r2) {
    if constexpr (NORMAL) {
        float r;
        asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(r2));
        return r;
    } else {
        return rsqrtf(r2);
    }
}

template <bool COMP, bool POT, bool STATS, int WARPS, bool NORMAL>
__global__ void __launch_bounds__(WARPS * 32, GBH_TRAVERSE_MIN_BLOCKS * kTravWarps / WARPS)
    k_traverse(
    const SimDesc* __restrict__ sims, const SimOut* __restrict__ simout,
    const uint32_t* __restrict__ chunk_sim, uint32_t nchunks, const float4* __restrict__ sbody,
    const CellRec* __restrict__ groups, const double4* __restrict__ cell_d, uint32_t capacity,
    unsigned long long* stats, uint32_t* err) {
    wait_for_predecessor();
    __shared__ uint2 s_stack[WARPS][kTravStack];  // (node group, lane mask)
    __shared__ float4 s_list[WARPS][kTravList];   // (com_x, com_y, G*m, lane mask bits)
    // mixed cells by rank: (lo bits, deciding lanes), the cell; f in list[32 + rank]
    __shared__ uint2 s_mix[WARPS][32];
    __shared__ uint32_t s_cell[WARPS][32];
    __shared__ uint32_t s_open[WARPS][32];  // the lanes that open them
    // compensated form: the f32 residual of each list entry's centre of mass
    // (0 for bodies), added back to the difference (com_hi - x) + com_lo, so a
    // term's distance carries the f64 centre of mass to one f32 rounding of
    // the distance itself rather than of the centre's coordinates
    __shared__ float2 s_lo[WARPS][COMP ? kTravList : 1];
    const uint32_t lane = lane_id();
    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t chunk = blockIdx.x * WARPS + warp;
    if (chunk >= nchunks) return;
    const uint32_t s = chunk_sim[chunk];
    if (s == kNone) return;
    const SimDesc& sd = sims[s];
    // each instance sums only the simulations that asked for its summation
    // form, so a simulation's forces do not depend on its batch mates
    if (((sd.flags & BH_FLAG_COMPENSATED) != 0u) != COMP) return;
    const uint32_t p0 = chunk * kChunk;
    const uint32_t p = p0 + lane;
    const bool valid = p < sd.off + sd.n;
    const float4 me = valid ? sbody[p] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float tx = me.x, ty = me.y;
    const float eps2 = sd.eps_f * sd.eps_f;
    const float g = sd.g_f;
    const uint32_t valid_mask = __ballot_sync(kFull, valid);
    const uint32_t lanes_below = (1u << lane) - 1u;
    float bx0 = valid ? tx : INFINITY, bx1 = valid ? tx : -INFINITY;
    float by0 = valid ? ty : INFINITY, by1 = valid ? ty : -INFINITY;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        bx0 = fminf(bx0, __shfl_xor_sync(kFull, bx0, o));
        bx1 = fmaxf(bx1, __shfl_xor_sync(kFull, bx1, o));
        by0 = fminf(by0, __shfl_xor_sync(kFull, by0, o));
        by1 = fmaxf(by1, __shfl_xor_sync(kFull, by1, o));
    }
    uint2* stack = s_stack[warp];
    float4* list = s_list[warp];
    Acc<COMP> acc;
    float phi = 0.f;
    uint32_t n_visit = 0, n_approx = 0, n_direct = 0, n_exact = 0, n_iter = 0;

    const float2 txy = make_float2(tx, ty);
    // one point-mass term at difference d, scale 0 for lanes that do not take it
    auto term = [&](float2 d, float d2, float gm, bool take) {
        const float inv_r = rsqrt_r2<NORMAL>(d2 + eps2);
        const float scale = take ? gm * inv_r * inv_r * inv_r : 0.f;
        acc.add_scaled(d, scale);
        if (POT) phi -= take ? gm * inv_r : 0.f;
    };
    const uint32_t lane_bit = 1u << lane;
    // A lane outside an entry's mask may sit at distance 0 from it (its own
    // body, with zero softening): its scale is selected to 0 after the
    // product, so the inf of that product never reaches the sums.
    auto flush = [&](uint32_t count) {
#pragma unroll 4
        for (uint32_t i = 0; i < count; ++i) {
            const float4 e = list[i];
            float2 d = sub2<COMP>(make_float2(e.x, e.y), txy);
            if constexpr (COMP) d = __fadd2_rn(d, s_lo[warp][i]);
            const float inv_r = rsqrt_r2<NORMAL>(__fmaf_rn(d.x, d.x, __fmaf_rn(d.y, d.y, eps2)));
            const bool take = (__float_as_uint(e.w) & lane_bit) != 0u;
            const float scale = e.z * inv_r * inv_r * inv_r;
            if constexpr (!COMP && !POT) {
                // plain sums: lanes outside the mask skip the (predicated) adds
                if (take) acc.add_scaled(d, scale);
            } else {
                acc.add_scaled(d, take ? scale : 0.f);
                if (POT) phi -= take ? e.z * inv_r : 0.f;
            }
        }
    };

    if (lane == 0) stack[0] = make_uint2(capacity + s, valid_mask);
    __syncwarp();
    uint32_t len = 1, nlist = 0;
    while (len > 0) {
        const uint32_t ng = min(len, 8u);
        const uint32_t gi = lane >> 2;
        const bool have = gi < ng;
        uint2 e = make_uint2(0u, 0u);
        if (have) e = stack[len - ng + gi];
        __syncwarp();
        len -= ng;
        float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
        uint4 u = make_uint4(0u, 0u, 0u, 0u);  // lo | count, start, count, cell (kNone: leaf)
        if (have) {
            const CellRec* r = groups + 4ull * e.x + (lane & 3u);
            f = __ldg(&r->f);
            u = __ldg(&r->u);
        }
        const uint32_t A = e.y;
        const bool present = u.z != 0u;
        const bool leaf = u.w == kNone;
        float2 clo = make_float2(0.f, 0.f);  // compensated: residual of the centre of mass
        if (COMP && have && present && !leaf) {
            const unsigned long long b = __double_as_longlong(
                __ldg(reinterpret_cast<const double*>(cell_d + u.w) + 3));
            clo = make_float2(__uint_as_float((uint32_t)b), __uint_as_float((uint32_t)(b >> 32)));
        }
        // lanes whose own body the cell holds: positions [start, start + count)
        const uint32_t ha = max(u.y, p0), hb = min(u.y + u.z, p0 + 32u);
        const uint32_t H = (present && ha < hb) ? bit_range(ha - p0, hb - p0) : 0u;
        const uint32_t R = A & ~H;
        // classification, branch-free (a select per outcome): a one-body
        // leaf is a list term for R; an internal cell is a list term for R
        // when the box's nearest point is beyond hi, opened by R when its
        // farthest corner is inside lo, otherwise mixed; holding lanes open it
        const float nx = fmaxf(fmaxf(bx0 - f.x, f.x - bx1), 0.f);
        const float ny = fmaxf(fmaxf(by0 - f.y, f.y - by1), 0.f);
        const float fx = fmaxf(fabsf(f.x - bx0), fabsf(f.x - bx1));
        const float fy = fmaxf(fabsf(f.y - by0), fabsf(f.y - by1));
        const bool internal = present && !leaf;
        const bool far = dist2(nx, ny) > f.w;
        const bool near = dist2(fx, fy) < __uint_as_float(u.x);
        const bool multi = present && leaf && u.z != 1u;
        const uint32_t ap = ((present && leaf && u.z == 1u) || (internal && far)) ? R : 0u;
        uint32_t op = internal ? ((A & H) | ((!far && near) ? R : 0u)) : 0u;
        const bool mixed = internal && R != 0u && !far && !near;
        if (STATS && present) {
            n_visit += __popc(A);
            if (leaf)
                n_direct += __popc(ap);
            else
                n_approx += __popc(ap);
        }
        if (STATS) ++n_iter;

        // mixed cells: every lane of the mask that does not hold the cell
        // decides for itself, one cell after the other; holding lanes open
        // it (op).  The record's f waits in the free upper half of the
        // interaction list (at most 31 entries are pending between steps),
        // the rest in s_mix and s_cell.  No branch in the loop (the lanes
        // inside a guard band come after it) and its results in an array it
        // does not read, so its turns overlap: 541 -> 513 us at 2^20 bodies,
        // 49 -> 40 at 2^14, 3608 -> 3447 at 2^22 compensated.
        const uint32_t bm = __ballot_sync(kFull, mixed);
        const uint32_t mrank = __popc(bm & lanes_below);
        if (mixed) {
            list[32u + mrank] = f;
            if (COMP) s_lo[warp][32u + mrank] = clo;
            s_mix[warp][mrank] = make_uint2(u.x, R);
            s_cell[warp][mrank] = u.w;
        }
        __syncwarp();
        const uint32_t nm = __popc(bm);
        uint32_t band = 0;  // the cells inside whose guard band this lane lies
#pragma unroll 4
        for (uint32_t i = 0; i < nm; ++i) {
            const float4 cf = list[32u + i];
            const uint2 cu = s_mix[warp][i];
            const bool active = (cu.y & lane_bit) != 0u;
            const float2 d = sub2<COMP>(make_float2(cf.x, cf.y), txy);
            const float d2 = dist2(d.x, d.y);
            const bool approx = active && d2 > cf.w;
            const bool open = active && d2 < __uint_as_float(cu.x);
            if (active && !approx && !open) band |= 1u << i;
            // branch-free: lanes that do not approximate add a zero term
            if constexpr (COMP) {
                const float2 dc = __fadd2_rn(d, s_lo[warp][32u + i]);
                term(dc, dist2(dc.x, dc.y), cf.z, approx);
            } else {
                term(d, d2, cf.z, approx);
            }
            if (STATS) n_approx += approx;
            const uint32_t O = __ballot_sync(kFull, open);
            if (lane == 0) s_open[warp][i] = O;
            if (STATS) ++n_iter;
        }
        // the lanes inside a guard band (a few in ten thousand decisions) decide
        // in f64 once the others are done
        for (uint32_t todo = __reduce_or_sync(kFull, band); todo != 0u; todo &= todo - 1u) {
            const uint32_t i = __ffs(todo) - 1u;
            const float4 cf = list[32u + i];
            const uint32_t cell = s_cell[warp][i];
            const bool mine = (band >> i) & 1u;
            const bool approx = mine && exact_mac(cell_d, cell, tx, ty, simout[s].half,
                                                  __float_as_uint(cf.w) & 31u, sd.theta);
            float2 d = sub2<COMP>(make_float2(cf.x, cf.y), txy);
            if constexpr (COMP) d = __fadd2_rn(d, s_lo[warp][32u + i]);
            term(d, dist2(d.x, d.y), cf.z, approx);
            if (STATS) {
                n_approx += approx;
                n_exact += mine;
            }
            const uint32_t O = __ballot_sync(kFull, mine && !approx);
            __syncwarp();
            if (lane == 0) s_open[warp][i] |= O;
        }
        __syncwarp();
        if (mixed) op |= s_open[warp][mrank];

        // leaves of several bodies: each body summed directly, self excluded
        uint32_t bl = __ballot_sync(kFull, multi);
        while (bl) {
            const uint32_t src = __ffs(bl) - 1u;
            bl &= bl - 1u;
            const uint32_t start = __shfl_sync(kFull, u.y, src);
            const uint32_t count = __shfl_sync(kFull, u.z, src);
            const uint32_t M = __shfl_sync(kFull, A, src);
            const bool active = (M >> lane) & 1u;
            for (uint32_t j = start; j < start + count; ++j) {
                const float4 o = sbody[j];
                const bool take = active && j != p;
                const float2 d = sub2<COMP>(make_float2(o.x, o.y), txy);
                term(d, dist2(d.x, d.y), __fmul_rn(g, o.z), take);
                if (STATS) n_direct += take;
            }
        }

        // append the uniform terms, push the opened groups in lane order
        const uint32_t la = __ballot_sync(kFull, ap != 0u);
        if (ap) {
            const uint32_t slot = nlist + __popc(la & lanes_below);
            list[slot] = make_float4(f.x, f.y, f.z, __uint_as_float(ap));
            if (COMP) s_lo[warp][slot] = clo;
        }
        nlist += __popc(la);
        const uint32_t lp = __ballot_sync(kFull, op != 0u);
        if (len + __popc(lp) > kTravStack) {  // unreachable by the bound above
            if (lane == 0) set_err(err, kErrTraversal);
            break;
        }
        if (op) stack[len + __popc(lp & lanes_below)] = make_uint2(u.w, op);
        len += __popc(lp);
        __syncwarp();
        if (nlist >= 32u) {
            flush(nlist);
            nlist = 0;
            __syncwarp();
        }
    }
    flush(nlist);
    if (valid) {
        const uint32_t idx = __float_as_uint(me.w);
        sd.accel[idx] = make_float4(acc.fx(), acc.fy(), 0.f, 0.f);
        if (POT && sd.potential) sd.potential[idx] = phi;
    }
    if (STATS) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            n_visit += __shfl_xor_sync(kFull, n_visit, o);
            n_approx += __shfl_xor_sync(kFull, n_approx, o);
            n_direct += __shfl_xor_sync(kFull, n_direct, o);
            n_exact += __shfl_xor_sync(kFull, n_exact, o);
        }
        if (lane == 0) {
            atomicAdd(&stats[0], (unsigned long long)n_visit);
            atomicAdd(&stats[1], (unsigned long long)n_approx);
            atomicAdd(&stats[2], (unsigned long long)n_direct);
            atomicAdd(&stats[3], (unsigned long long)n_exact);
            atomicAdd(&stats[4], (unsigned long long)n_iter);
        }
    }
}

// ======================================================== packed (2B1) ====

// runtime/src/nbody.wgsl:43-123 (and barnes_hut_flat.cu:65-146) over an
// arbitrary packed tree with explicit children: the same per-body decisions
// (f32 MAC with sqrt), self-exclusion and terms, computed for a warp of 32
// consecutive Morton positions at once.
constexpr int kPackedStack = 64;

__device__ __forceinline__ void packed_point_mass(float tx, float ty, float px, float py,
                                                  float mass, float soft, float g, float* ax,
                                                  float* ay) {
    const float dx = px - tx;
    const float dy = py - ty;
    const float r2 = dx * dx + dy * dy + soft * soft;
    const float inv_r = rsqrtf(r2);
    const float scale = g * mass * inv_r * inv_r * inv_r;
    *ax += dx * scale;
    *ay += dy * scale;
}

// Whether every position's entry names a body whose recorded Morton
// position is that position (bodies[entries[p].body].meta[0] == p), i.e. the
// entries are a permutation of the bodies and meta its inverse, as
// pack_flat_tree writes them.  *bad gets 1 otherwise.  The lane-parallel
// walk relies on it: a lane's own body is the one at its position.
__global__ void k_check_packed(const GpuBody* __restrict__ bodies,
                               const GpuEntry* __restrict__ entries, uint32_t n, uint32_t* bad) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const uint32_t o = entries[p].data[1];
    if (o >= n || bodies[o].meta[0] != p) atomicOr(bad, 1u);
}

// The walk one cell at a time: every lane of the warp tests the same cell
// and keeps the reference's depth-first order of its own terms (children
// pushed 3..0).  Used when the entries and bodies disagree or a tree is
// deeper than the lane-parallel walk's stack bound.  s_cell / s_mask hold
// kPackedStack entries each.
__device__ void packed_walk_cellwise(const BhSettings& st, const GpuBody* __restrict__ bodies,
                                     const GpuEntry* __restrict__ entries,
                                     const GpuCell* __restrict__ cells, uint32_t n,
                                     uint32_t ncells, uint32_t ti, float tx, float ty,
                                     uint32_t tpos, bool lane_ok, uint32_t* s_cell,
                                     uint32_t* s_mask, uint32_t* err, float* out_ax,
                                     float* out_ay) {
    const float theta = st.physics[0], soft = st.physics[1], g = st.physics[2];
    const uint32_t lane = lane_id();
    float ax = 0.f, ay = 0.f;
    int len = 1;
    const uint32_t vmask = __ballot_sync(kFull, lane_ok);
    if (lane == 0) {
        s_cell[0] = st.info[2];
        s_mask[0] = vmask;
    }
    __syncwarp();
    while (len > 0) {
        --len;
        const uint32_t ci = s_cell[len];
        const uint32_t M = s_mask[len];
        __syncwarp();
        if (ci >= ncells) {
            set_err(err, kErrPackedIndex);
            break;
        }
        const GpuCell cell = cells[ci];
        const bool active = (M >> lane) & 1u;
        const bool leaf = cell.children[0] == GALAXY_BH_NO_CHILD &&
                          cell.children[1] == GALAXY_BH_NO_CHILD &&
                          cell.children[2] == GALAXY_BH_NO_CHILD &&
                          cell.children[3] == GALAXY_BH_NO_CHILD;
        if (leaf) {
            for (uint32_t q = cell.range_depth[0]; q < cell.range_depth[1]; ++q) {
                if (q >= n) {
                    set_err(err, kErrPackedIndex);
                    break;
                }
                const uint32_t o = entries[q].data[1];
                if (active && o != ti && o < n) {
                    const GpuBody ob = bodies[o];
                    packed_point_mass(tx, ty, ob.position_mass[0], ob.position_mass[1],
                                      ob.position_mass[2], soft, g, &ax, &ay);
                }
            }
            continue;
        }
        bool open = false;
        if (active) {
            const float dx = cell.com[0] - tx;
            const float dy = cell.com[1] - ty;
            const float distance2 = dx * dx + dy * dy;
            const bool contains = tpos >= cell.range_depth[0] && tpos < cell.range_depth[1];
            open = true;
            if (!contains && distance2 > 0.0f) {
                const float distance = sqrtf(distance2);
                if ((2.0f * cell.center_half_mass[2]) / distance < theta) {
                    packed_point_mass(tx, ty, cell.com[0], cell.com[1], cell.center_half_mass[3],
                                      soft, g, &ax, &ay);
                    open = false;
                }
            }
        }
        const uint32_t O = __ballot_sync(kFull, open);
        if (O) {
            int nch = 0;
#pragma unroll
            for (int q = 0; q < 4; ++q) nch += cell.children[q] != GALAXY_BH_NO_CHILD;
            if (len + nch > kPackedStack) {
                set_err(err, kErrPackedStack);
                break;
            }
            if (lane == 0) {
                for (int q = 3; q >= 0; --q) {
                    if (cell.children[q] != GALAXY_BH_NO_CHILD) {
                        s_cell[len] = cell.children[q];
                        s_mask[len] = O;
                        ++len;
                    }
                }
            }
            len = __shfl_sync(kFull, len, 0);
            __syncwarp();
        }
    }
    *out_ax = ax;
    *out_ay = ay;
}

// Lane-parallel walk over the packed tree, the structure of k_traverse: a
// warp pops up to 8 opened cells from its shared-memory stack and lane 4i+q
// examines child q of popped cell i for all lanes of its mask at once,
// against the bounding box of the warp's bodies.  The reference decides in
// f32: a lane approximates a cell unless the cell holds its own body, if
// its squared distance d2 to the centre of mass is positive and
// (2 half) / sqrt(d2) < theta.  d2 = fma(dx, dx, dy*dy), sqrt and the
// division are monotone in |dx|, |dy| (round to nearest), so the test at
// the box's nearest point (all lanes approximate) or farthest corner (all
// open) is every lane's own test; other cells are decided lane by lane
// with the same expression.  Approximated cells and one-body leaves go to
// the interaction list, several-body leaves are summed body by body; a
// lane's own body is the one at its position (the entries are checked to be
// a permutation whose inverse the bodies record), so self-exclusion is
// the lane bit of that position.  Each lane sums exactly the reference's
// terms; only their order differs.
constexpr uint32_t kPkWarps = 4;
constexpr uint32_t kPkRoot = 0xfffffffeu;  // stack entry standing for the root cell itself
// (cell, lane mask) entries: the stack stays sorted by depth and one step
// pushes at most 32 opened cells, so 32 per level of a tree of depth 16
// (pack_flat_tree's trees); a deeper tree that overflows it is walked again
// cell by cell
constexpr uint32_t kPkStack = 17u * 32u;
static_assert(2u * kPkStack >= 2u * kPackedStack, "the cell-by-cell walk borrows the stack");

__global__ void __launch_bounds__(kPkWarps * 32) k_traverse_packed(
    const BhSettings* __restrict__ settings, const GpuBody* __restrict__ bodies,
    const GpuEntry* __restrict__ entries, const GpuCell* __restrict__ cells, uint32_t n,
    uint32_t ncells, float4* __restrict__ accel, uint32_t* err,
    const uint32_t* __restrict__ inconsistent) {
    __shared__ uint2 s_stack[kPkWarps][kPkStack];
    __shared__ float4 s_list[kPkWarps][kTravList];  // (x, y, G*m, lane mask bits)
    __shared__ uint32_t s_mix[kPkWarps][32][2];      // mixed cells by rank: deciding, opened
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    const uint32_t p0 = (blockIdx.x * kPkWarps + warp) * 32u;
    if (p0 >= n) return;
    const BhSettings st = *settings;
    const float theta = st.physics[0], soft = st.physics[1], g = st.physics[2];
    const uint32_t p = p0 + lane;
    const bool valid = p < n;
    uint32_t* s_cell = reinterpret_cast<uint32_t*>(s_stack[warp]);
    float ax = 0.f, ay = 0.f;
    if (*inconsistent) {
        // the reference's own indexing: lane p walks for body p, at the
        // Morton position that body records
        const GpuBody b = valid ? bodies[p] : GpuBody{};
        packed_walk_cellwise(st, bodies, entries, cells, n, ncells, p, b.position_mass[0],
                             b.position_mass[1], b.meta[0], valid, s_cell,
                             s_cell + kPackedStack, err, &ax, &ay);
        if (valid) accel[p] = make_float4(ax, ay, 0.f, 0.f);
        return;
    }
    // consistent input: the body at position p is ti, and it records p
    const uint32_t ti = valid ? entries[p].data[1] : 0u;
    const GpuBody tb = valid ? bodies[ti] : GpuBody{};
    const float tx = tb.position_mass[0], ty = tb.position_mass[1];
    const float eps2 = soft * soft;
    const uint32_t valid_mask = __ballot_sync(kFull, valid);
    const uint32_t lanes_below = (1u << lane) - 1u;
    const uint32_t lane_bit = 1u << lane;
    float bx0 = valid ? tx : INFINITY, bx1 = valid ? tx : -INFINITY;
    float by0 = valid ? ty : INFINITY, by1 = valid ? ty : -INFINITY;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        bx0 = fminf(bx0, __shfl_xor_sync(kFull, bx0, o));
        bx1 = fmaxf(bx1, __shfl_xor_sync(kFull, bx1, o));
        by0 = fminf(by0, __shfl_xor_sync(kFull, by0, o));
        by1 = fmaxf(by1, __shfl_xor_sync(kFull, by1, o));
    }
    uint2* stack = s_stack[warp];
    float4* list = s_list[warp];
    // one point-mass term (the reference's add_point_mass) for lanes that take it
    auto term = [&](float dx, float dy, float gm, bool take) {
        const float inv_r = rsqrtf(__fmaf_rn(dx, dx, __fmaf_rn(dy, dy, eps2)));
        const float scale = gm * inv_r * inv_r * inv_r;
        if (take) {
            ax += dx * scale;
            ay += dy * scale;
        }
    };
    auto flush = [&](uint32_t count) {
#pragma unroll 4
        for (uint32_t i = 0; i < count; ++i) {
            const float4 e = list[i];
            term(e.x - tx, e.y - ty, e.z, (__float_as_uint(e.w) & lane_bit) != 0u);
        }
    };
    // the reference's opening test: true = approximate
    auto approximates = [&](float two_half, float d2) {
        return d2 > 0.0f && two_half / sqrtf(d2) < theta;
    };

    if (lane == 0) stack[0] = make_uint2(kPkRoot, valid_mask);
    __syncwarp();
    uint32_t len = 1, nlist = 0;
    bool overflow = false;
    while (len > 0) {
        const uint32_t ng = min(len, 8u);
        const uint32_t gi = lane >> 2, q = lane & 3u;
        const bool have = gi < ng;
        uint2 e = make_uint2(0u, 0u);
        if (have) e = stack[len - ng + gi];
        __syncwarp();
        len -= ng;
        uint32_t c = GALAXY_BH_NO_CHILD;
        if (have) c = e.x == kPkRoot ? (q == 0u ? st.info[2] : GALAXY_BH_NO_CHILD)
                                     : __ldg(&cells[e.x].children[q]);
        bool present = c != GALAXY_BH_NO_CHILD;
        if (present && c >= ncells) {
            set_err(err, kErrPackedIndex);
            present = false;
        }
        float4 chm = make_float4(0.f, 0.f, 0.f, 0.f);  // centre, half, mass
        float2 com = make_float2(0.f, 0.f);
        uint4 rd = make_uint4(0u, 0u, 0u, 0u);          // start, end, depth, valid
        uint4 chn = make_uint4(GALAXY_BH_NO_CHILD, GALAXY_BH_NO_CHILD, GALAXY_BH_NO_CHILD,
                               GALAXY_BH_NO_CHILD);
        if (present) {
            const GpuCell* cr = cells + c;
            chm = __ldg(reinterpret_cast<const float4*>(cr->center_half_mass));
            com = __ldg(reinterpret_cast<const float2*>(cr->com));
            rd = __ldg(reinterpret_cast<const uint4*>(cr->range_depth));
            chn = __ldg(reinterpret_cast<const uint4*>(cr->children));
        }
        const uint32_t A = e.y;
        const bool leaf = chn.x == GALAXY_BH_NO_CHILD && chn.y == GALAXY_BH_NO_CHILD &&
                          chn.z == GALAXY_BH_NO_CHILD && chn.w == GALAXY_BH_NO_CHILD;
        // lanes whose own body the cell holds: positions [start, end)
        const uint32_t ha = max(rd.x, p0), hb = min(rd.y, p0 + 32u);
        const uint32_t H = (present && ha < hb) ? bit_range(ha - p0, hb - p0) : 0u;
        const uint32_t R = A & ~H;
        const bool internal = present && !leaf;
        const bool one = present && leaf && rd.y == rd.x + 1u;
        const bool multi = present && leaf && rd.y > rd.x + 1u;
        // a one-body leaf is a term at its body (the reference sums leaves
        // from the bodies themselves)
        float ex = com.x, ey = com.y, em = chm.w;
        if (one) {
            if (rd.x < n) {
                const float4 b = __ldg(reinterpret_cast<const float4*>(
                    bodies[__ldg(&entries[rd.x].data[1])].position_mass));
                ex = b.x;
                ey = b.y;
                em = b.z;
            } else {
                set_err(err, kErrPackedIndex);
            }
        }
        const float two_half = 2.0f * chm.z;
        const float nx = fmaxf(fmaxf(bx0 - com.x, com.x - bx1), 0.f);
        const float ny = fmaxf(fmaxf(by0 - com.y, com.y - by1), 0.f);
        const float fx = fmaxf(fabsf(com.x - bx0), fabsf(com.x - bx1));
        const float fy = fmaxf(fabsf(com.y - by0), fabsf(com.y - by1));
        const bool far = internal && approximates(two_half, dist2(nx, ny));
        const bool near = internal && !approximates(two_half, dist2(fx, fy));
        const uint32_t ap = (one || far) ? R : 0u;
        uint32_t op = internal ? ((A & H) | (near ? R : 0u)) : 0u;
        const bool mixed = internal && R != 0u && !far && !near;

        // mixed cells: every lane of the mask that does not hold the cell
        // decides for itself, one cell after the other, from a copy of the
        // cell parked in the free upper half of the interaction list
        const uint32_t bm = __ballot_sync(kFull, mixed);
        const uint32_t mrank = __popc(bm & lanes_below);
        if (mixed) {
            list[32u + mrank] = make_float4(com.x, com.y, g * chm.w, two_half);
            s_mix[warp][mrank][0] = R;
        }
        __syncwarp();
        const uint32_t nm = __popc(bm);
        for (uint32_t i = 0; i < nm; ++i) {
            const float4 cf = list[32u + i];
            const bool active = (s_mix[warp][i][0] & lane_bit) != 0u;
            const float dx = cf.x - tx, dy = cf.y - ty;
            const bool approx = active && approximates(cf.w, dist2(dx, dy));
            term(dx, dy, cf.z, approx);
            const uint32_t O = __ballot_sync(kFull, active && !approx);
            if (lane == 0) s_mix[warp][i][1] = O;
        }
        __syncwarp();
        if (mixed) op |= s_mix[warp][mrank][1];

        // leaves of several bodies: each body summed directly, self excluded
        uint32_t bl = __ballot_sync(kFull, multi);
        while (bl) {
            const uint32_t src = __ffs(bl) - 1u;
            bl &= bl - 1u;
            const uint32_t start = __shfl_sync(kFull, rd.x, src);
            const uint32_t end = __shfl_sync(kFull, rd.y, src);
            const uint32_t M = __shfl_sync(kFull, A, src);
            const bool active = (M >> lane) & 1u;
            if (end > n) set_err(err, kErrPackedIndex);
            for (uint32_t j = start; j < min(end, n); ++j) {
                const float4 b = __ldg(reinterpret_cast<const float4*>(
                    bodies[__ldg(&entries[j].data[1])].position_mass));
                term(b.x - tx, b.y - ty, g * b.z, active && j != p);
            }
        }

        // append the list terms, push the opened cells in lane order
        const uint32_t la = __ballot_sync(kFull, ap != 0u);
        if (ap) list[nlist + __popc(la & lanes_below)] = make_float4(ex, ey, g * em,
                                                                      __uint_as_float(ap));
        nlist += __popc(la);
        const uint32_t lp = __ballot_sync(kFull, op != 0u);
        if (len + __popc(lp) > kPkStack) {  // deeper than the bound: walk again cell by cell
            overflow = true;
            break;
        }
        if (op) stack[len + __popc(lp & lanes_below)] = make_uint2(c, op);
        len += __popc(lp);
        __syncwarp();
        if (nlist >= 32u) {
            flush(nlist);
            nlist = 0;
            __syncwarp();
        }
    }
    if (overflow) {
        __syncwarp();
        packed_walk_cellwise(st, bodies, entries, cells, n, ncells, ti, tx, ty, p, valid, s_cell,
                             s_cell + kPackedStack, err, &ax, &ay);
    } else {
        flush(nlist);
    }
    if (valid) accel[ti] = make_float4(ax, ay, 0.f, 0.f);
}

// ============================================================ export =====

// Frozen 64-byte cells (pack_flat_tree, nbody_gpu.rs:211-229) of one
// simulation in the reference preorder, plus sorted entries and bodies with
// their Morton positions.  Cell centres are rebuilt from the code prefix
// with the same f64 steps as child_bounds (nbody/src/flat.rs:96-103).
__global__ void k_export_cells(const SimDesc* __restrict__ sims, const SimOut* __restrict__ simout,
                               uint32_t sim, const uint32_t* __restrict__ codes,
                               const uint32_t* __restrict__ base,
                               const uint4* __restrict__ cell_u,
                               const double4* __restrict__ cell_d, GpuCell* out) {
    const SimDesc& sd = sims[sim];
    const uint32_t cb = base[sd.off], ce = base[sd.off + sd.n];
    const uint32_t k = cb + blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= ce) return;
    const SimOut so = simout[sim];
    const uint4 u = cell_u[k];
    const uint32_t start = u.z - sd.off;
    const uint32_t code = codes[u.z];
    double cx = so.cx, cy = so.cy, half = so.half;
    for (uint32_t level = 0; level < u.w; ++level) {
        const uint32_t q = (code >> (30u - 2u * level)) & 3u;
        const double h = __dmul_rn(half, 0.5);
        cx = __dadd_rn(cx, (q & 1u) ? h : -h);
        cy = __dadd_rn(cy, (q & 2u) ? h : -h);
        half = h;
    }
    const double4 v = cell_d[k];
    GpuCell c;
    c.center_half_mass[0] = (float)cx;
    c.center_half_mass[1] = (float)cy;
    c.center_half_mass[2] = (float)half;
    c.center_half_mass[3] = (float)v.z;
    c.com[0] = (float)v.x;
    c.com[1] = (float)v.y;
    c.com[2] = 0.f;
    c.com[3] = 0.f;
    c.range_depth[0] = start;
    c.range_depth[1] = u.x - sd.off;
    c.range_depth[2] = u.w;
    c.range_depth[3] = 0u;
    // children: k + 1, then each at the one before's skip (none for a leaf)
    uint32_t child[4] = {kNone, kNone, kNone, kNone};
    for (uint32_t next = k + 1u; next < u.y;) {
        const uint4 cu = cell_u[next];
        const uint32_t quadrant = (codes[cu.z] >> (30u - 2u * u.w)) & 3u;
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q) child[q] = q == quadrant ? next - cb : child[q];
        next = cu.y;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) c.children[q] = child[q];
    out[k - cb] = c;
}

__global__ void k_export_entries(const SimDesc* __restrict__ sims, uint32_t sim,
                                 const uint32_t* __restrict__ codes,
                                 const float4* __restrict__ sbody, GpuEntry* entries,
                                 GpuBody* bodies) {
    const SimDesc& sd = sims[sim];
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= sd.n) return;
    const float4 b = sbody[sd.off + i];
    const uint32_t idx = __float_as_uint(b.w);
    if (entries) {
        GpuEntry e;
        e.data[0] = codes[sd.off + i];
        e.data[1] = idx;
        e.data[2] = 0u;
        e.data[3] = 0u;
        entries[i] = e;
    }
    if (bodies) {
        GpuBody gb;
        gb.position_mass[0] = b.x;
        gb.position_mass[1] = b.y;
        gb.position_mass[2] = b.z;
        gb.position_mass[3] = 0.f;
        gb.meta[0] = i;
        gb.meta[1] = gb.meta[2] = gb.meta[3] = 0u;
        bodies[idx] = gb;
    }
}

// ===================================================== direct probes =====

constexpr int kProbeThreads = 256;
constexpr int kProbesPerBlock = 8;

// FP64 direct sums for probe bodies (direct_acceleration_for,
// nbody/src/lib.rs:315-329, over the f32 state promoted to f64): every term
// is that of nbody/src/lib.rs:247-255 in f64, with the reciprocal square root and
// fused multiply-adds where the reference divides 1 by a square root and rounds
// each product: the root is within 1 ulp and enters three times, so a term differs
// by a few ulp.  Each thread sums a strided share of a slice of the sources, the
// block adds the shares in a fixed order and k_add_slices the slices.  The slices
// (grid.y) fill the chip whatever the number of probes: with every source in one block
// 4,096 probes were 512 blocks, 1.15 waves of the 444 resident ones, and 12
// probes 2 blocks; 4,096 probes of 2^20 bodies, a whole call, 16.3 -> 10.0 ms.
// The f64 pipe bounds it: with rsqrt for a square root and a division 9.1 -> 5.4 ms.
// Errors against sums in 80 bits, relative to the result (median of 100 to 400
// probes): 2^20 bodies 5.5e-17 (2.3e-16 with the sources in one block, rounded
// products and a division), 262,147 5.7e-17 (1.7e-16), 4,099 1.5e-16 (1.5e-16).
__global__ void __launch_bounds__(kProbeThreads) k_direct_probes(
    const GpuEvolveState* __restrict__ state, uint32_t n, const uint32_t* __restrict__ probes,
    uint32_t nprobes, uint32_t slice, double eps, double g, double* __restrict__ out) {
    __shared__ double sh[kProbesPerBlock][2][kProbeThreads];
    double tx[kProbesPerBlock], ty[kProbesPerBlock], ax[kProbesPerBlock], ay[kProbesPerBlock];
    uint32_t ti[kProbesPerBlock];
#pragma unroll
    for (int k = 0; k < kProbesPerBlock; ++k) {
        const uint32_t q = blockIdx.x * kProbesPerBlock + k;
        ti[k] = q < nprobes ? probes[q] : kNone;
        const bool ok = ti[k] < n;
        tx[k] = ok ? (double)state[ti[k]].position_mass[0] : 0.0;
        ty[k] = ok ? (double)state[ti[k]].position_mass[1] : 0.0;
        ax[k] = ay[k] = 0.0;
    }
    const double eps2 = __dmul_rn(eps, eps);
    const uint32_t end = min(n - blockIdx.y * slice, slice) + blockIdx.y * slice;
    for (uint32_t j = blockIdx.y * slice + threadIdx.x; j < end; j += kProbeThreads) {
        const float4 pm = *reinterpret_cast<const float4*>(state + j);
        const double x = pm.x, y = pm.y, m = pm.z;
        const double gm = __dmul_rn(g, m);
#pragma unroll
        for (int k = 0; k < kProbesPerBlock; ++k) {
            if (j == ti[k]) continue;
            const double dx = __dsub_rn(x, tx[k]);
            const double dy = __dsub_rn(y, ty[k]);
            const double inv_r = rsqrt(__fma_rn(dx, dx, __fma_rn(dy, dy, eps2)));
            const double scale = __dmul_rn(__dmul_rn(__dmul_rn(gm, inv_r), inv_r), inv_r);
            ax[k] = __fma_rn(dx, scale, ax[k]);
            ay[k] = __fma_rn(dy, scale, ay[k]);
        }
    }
#pragma unroll
    for (int k = 0; k < kProbesPerBlock; ++k) {
        sh[k][0][threadIdx.x] = ax[k];
        sh[k][1][threadIdx.x] = ay[k];
    }
    __syncthreads();
    for (int stride = kProbeThreads / 2; stride > 0; stride >>= 1) {
        if ((int)threadIdx.x < stride)
#pragma unroll
            for (int k = 0; k < kProbesPerBlock; ++k) {
                sh[k][0][threadIdx.x] += sh[k][0][threadIdx.x + stride];
                sh[k][1][threadIdx.x] += sh[k][1][threadIdx.x + stride];
            }
        __syncthreads();
    }
    if (threadIdx.x < kProbesPerBlock) {
        const uint32_t q = blockIdx.x * kProbesPerBlock + threadIdx.x;
        if (q < nprobes) {
            double* slot = out + 2 * ((size_t)blockIdx.y * nprobes + q);
            slot[0] = sh[threadIdx.x][0][0];
            slot[1] = sh[threadIdx.x][1][0];
        }
    }
}

// out[i] = the sum of the slices' values, in slice order; values[0] may be out.
// There are up to 4,440 (512 with few probes of 2^20 bodies, 2,048 of 2^22), and one
// after the other already 512 cost more than the rest of the sum together (6e-16
// against 4e-16 of the result), so each addition's rounding is kept and added at the
// end (Knuth's two-sum).
__global__ void __launch_bounds__(256) k_add_slices(const double* values, uint32_t count,
                                                    uint32_t slices, double* out) {
    const uint32_t i = blockIdx.x * 256u + threadIdx.x;
    if (i >= count) return;
    double sum = values[i], rest = 0.0;
    for (uint32_t k = 1; k < slices; ++k) {
        const double v = values[(size_t)k * count + i];
        const double t = __dadd_rn(sum, v), b = __dsub_rn(t, sum);
        rest = __dadd_rn(rest, __dadd_rn(__dsub_rn(sum, __dsub_rn(t, b)), __dsub_rn(v, b)));
        sum = t;
    }
    // (an infinite or NaN sum has no rest)
    out[i] = isfinite(sum) ? __dadd_rn(sum, rest) : sum;
}

// Slices of the sources: enough blocks for about ten waves (a last one that is
// nearly empty then costs little), of at least 2,048 sources each.
uint32_t probe_slices(uint32_t n, uint32_t nprobes) {
    const uint64_t blocks = (nprobes + kProbesPerBlock - 1ull) / kProbesPerBlock;
    const uint64_t want = 4440ull / blocks, most = (n + 2047ull) / 2048ull;
    const uint64_t slices = want < most ? want : most;
    return slices ? (uint32_t)slices : 1u;
}

cudaError_t launch_direct_probes(const GpuEvolveState* state, uint32_t n, const uint32_t* probes,
                                 uint32_t nprobes, double eps, double g, double* out,
                                 cudaStream_t s) {
    const uint32_t blocks = (nprobes + kProbesPerBlock - 1) / kProbesPerBlock;
    const uint32_t want = probe_slices(n, nprobes);
    const uint32_t slice = (n + want - 1) / want, slices = (n + slice - 1) / slice;
    k_direct_probes<<<dim3(blocks, slices), kProbeThreads, 0, s>>>(state, n, probes, nprobes, slice,
                                                                  eps, g, out);
    if (slices > 1)
        k_add_slices<<<(2 * nprobes + 255) / 256, 256, 0, s>>>(out, 2 * nprobes, slices, out);
    return cudaGetLastError();
}

// ================================================= f64 flat traversal =====

// The reference CPU flat traversal (flat_acceleration_for,
// nbody/src/flat.rs:270-346) in f64 over this engine's tree, one thread per
// body in Morton order.  The cells are numbered in the reference's preorder,
// so its depth-first stack walk (children pushed 3..0, popped 0 first) is
// the walk k -> k + 1 when a cell opens and k -> skip when a leaf is summed
// or a cell approximated: each body meets the same cells in the same order,
// with the same f64 centres of mass and masses (bit-identical aggregates),
// the same MAC (hypot distance, width / distance < theta, a cell holding the
// body always opens) and the per-term arithmetic of nbody/src/lib.rs:247-255
// as explicit round-to-nearest operations, so the sum repeats the
// reference's additions one for one.  abs_sum (optional) gets the sum of
// the terms' magnitudes |G m d / r^3| per body; stats the reference's force
// counters (visited, approximated, direct).
constexpr int kF64Threads = 128;

__global__ void __launch_bounds__(kF64Threads) k_traverse_f64(
    const SimDesc* __restrict__ sims, const SimOut* __restrict__ simout, uint32_t sim,
    const float4* __restrict__ sbody, const uint4* __restrict__ cell_u,
    const double4* __restrict__ cell_d, const uint32_t* __restrict__ base, double theta,
    double eps, double g, double2* __restrict__ out, double* __restrict__ abs_sum,
    unsigned long long* __restrict__ stats) {
    const SimDesc& sd = sims[sim];
    const uint32_t i = blockIdx.x * kF64Threads + threadIdx.x;
    unsigned long long nv = 0, na = 0, nd = 0;
    if (i < sd.n) {
        const uint32_t p = sd.off + i;
        const float4 me = sbody[p];
        const double tx = me.x, ty = me.y;
        const double eps2 = __dmul_rn(eps, eps);
        const double root_half = simout[sim].half;
        double ax = 0.0, ay = 0.0, s = 0.0;
        auto add = [&](double x, double y, double mass) {
            const double dx = __dsub_rn(x, tx);
            const double dy = __dsub_rn(y, ty);
            const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), eps2);
            const double inv_r = __ddiv_rn(1.0, __dsqrt_rn(r2));
            const double scale =
                __dmul_rn(__dmul_rn(__dmul_rn(__dmul_rn(g, mass), inv_r), inv_r), inv_r);
            const double fx = __dmul_rn(dx, scale), fy = __dmul_rn(dy, scale);
            ax = __dadd_rn(ax, fx);
            ay = __dadd_rn(ay, fy);
            if (abs_sum) s += hypot(fx, fy);
        };
        const uint32_t root = base[sd.off];
        const uint32_t stop = cell_u[root].y;  // the root's skip: past the last cell
        uint32_t k = root;
        while (k < stop) {
            const uint4 u = cell_u[k];  // (end, skip, start, depth)
            ++nv;
            if (u.y == k + 1u) {  // a leaf: its bodies directly, self excluded
                for (uint32_t q = u.z; q < u.x; ++q) {
                    if (q == p) continue;
                    const float4 o = sbody[q];
                    add((double)o.x, (double)o.y, (double)o.z);
                    ++nd;
                }
                k = u.y;
                continue;
            }
            const double4 c = cell_d[k];
            const double dist = hypot(__dsub_rn(c.x, tx), __dsub_rn(c.y, ty));
            const double width = __dmul_rn(__dmul_rn(root_half, pow2_neg(u.w)), 2.0);
            const bool contains = p >= u.z && p < u.x;
            if (!contains && dist > 0.0 && __ddiv_rn(width, dist) < theta) {
                add(c.x, c.y, c.z);
                ++na;
                k = u.y;
            } else {
                k = k + 1u;  // open: the first child follows its parent
            }
        }
        const uint32_t idx = __float_as_uint(me.w);
        out[idx] = make_double2(ax, ay);
        if (abs_sum) abs_sum[idx] = s;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        nv += __shfl_xor_sync(kFull, nv, o);
        na += __shfl_xor_sync(kFull, na, o);
        nd += __shfl_xor_sync(kFull, nd, o);
    }
    if (stats && lane_id() == 0 && nv) {
        atomicAdd(&stats[0], nv);
        atomicAdd(&stats[1], na);
        atomicAdd(&stats[2], nd);
    }
}

cudaError_t launch_traverse_f64(const BatchBuffers& b, uint32_t sim, uint32_t n, double theta,
                                double eps, double g, double* out, double* abs_sum,
                                unsigned long long* stats, cudaStream_t s) {
    const uint32_t blocks = (n + kF64Threads - 1) / kF64Threads;
    if (blocks == 0) return cudaSuccess;
    k_traverse_f64<<<blocks, kF64Threads, 0, s>>>(b.sims, b.simout, sim, b.sbody, b.cell_u,
                                                  b.cell_d, b.base, theta, eps, g,
                                                  reinterpret_cast<double2*>(out), abs_sum, stats);
    return cudaGetLastError();
}

// ======================================================= conservation =====

constexpr int kConsThreads = 256;
constexpr int kConsTerms = 9;

// Per-block f64 partial sums in a fixed order, then one block adds the
// partials, a warp per term, in a fixed order: the result does not depend on
// scheduling.
__global__ void __launch_bounds__(kConsThreads) k_conservation_partial(
    const GpuEvolveState* __restrict__ state, const float* __restrict__ potential, uint32_t n,
    double* partials) {
    __shared__ double sh[kConsTerms][kConsThreads];
    double t[kConsTerms] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    for (uint32_t i = blockIdx.x * kConsThreads + threadIdx.x; i < n;
         i += gridDim.x * kConsThreads) {
        const GpuEvolveState s = state[i];
        const double m = s.position_mass[2], x = s.position_mass[0], y = s.position_mass[1];
        const double vx = s.velocity[0], vy = s.velocity[1];
        t[0] += m;
        t[1] += m * x;
        t[2] += m * y;
        t[3] += m * vx;
        t[4] += m * vy;
        t[5] += m * (x * vy - y * vx);
        t[6] += 0.5 * m * (vx * vx + vy * vy);
        if (potential) t[7] += 0.5 * m * (double)potential[i];
        t[8] += m * hypot(vx, vy);
    }
#pragma unroll
    for (int k = 0; k < kConsTerms; ++k) sh[k][threadIdx.x] = t[k];
    __syncthreads();
    for (int stride = kConsThreads / 2; stride > 0; stride >>= 1) {
        if ((int)threadIdx.x < stride)
#pragma unroll
            for (int k = 0; k < kConsTerms; ++k) sh[k][threadIdx.x] += sh[k][threadIdx.x + stride];
        __syncthreads();
    }
    if (threadIdx.x < kConsTerms) partials[blockIdx.x * kConsTerms + threadIdx.x] = sh[threadIdx.x][0];
}

// A warp per term: lane l adds partials l, l + 32, ..., the lanes pairwise.  (One
// thread per term was a chain of 592 additions behind their loads: a call at
// 262,147 bodies 51 -> 36 us, at 2^22 83 -> 53.)
__global__ void __launch_bounds__(32 * kConsTerms) k_conservation_final(
    const double* __restrict__ partials, uint32_t nblocks, double* out) {
    const uint32_t term = threadIdx.x >> 5;
    double acc = 0.0;
    for (uint32_t b = lane_id(); b < nblocks; b += 32u) acc += partials[b * kConsTerms + term];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(kFull, acc, o);
    if (lane_id() == 0) out[term] = acc;
}

// ============================================================ launchers ===

static int sm_count();

// One resident wave of integrate blocks (each warp then streams a contiguous
// run of chunks), fewer when there are fewer chunks than warps.
template <int MODE>
static uint32_t integrate_blocks(uint32_t nchunks) {
    static int per_sm[64] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    int& r = per_sm[dev & 63];
    if (!r) {
        int v = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, k_integrate<MODE>, 256, 0);
        r = v > 0 ? v : 1;
    }
#ifdef GBH_INTEGRATE_BLOCKS_PER_SM
    const uint32_t cap = (uint32_t)(sm_count() * GBH_INTEGRATE_BLOCKS_PER_SM);
#else
    // the final kick (no bounds atomics): one warp per chunk
    const uint32_t cap = MODE == 2 ? 0xffffffffu : (uint32_t)(sm_count() * r);
#endif
    const uint32_t blocks = (nchunks + 7) / 8;
    return blocks < cap ? (blocks ? blocks : 1u) : cap;
}

cudaError_t launch_integrate(const BatchBuffers& b, int mode, cudaStream_t s) {
    switch (mode) {
        case 0: return launch_step(k_integrate<0>, integrate_blocks<0>(b.nchunks), 256, 0, s, b.sims, b.chunk_sim, b.nchunks, b.minmax);
        case 1: return launch_step(k_integrate<1>, integrate_blocks<1>(b.nchunks), 256, 0, s, b.sims, b.chunk_sim, b.nchunks, b.minmax);
        case 2: return launch_step(k_integrate<2>, integrate_blocks<2>(b.nchunks), 256, 0, s, b.sims, b.chunk_sim, b.nchunks, b.minmax);
        default: return launch_step(k_integrate<3>, integrate_blocks<3>(b.nchunks), 256, 0, s, b.sims, b.chunk_sim, b.nchunks, b.minmax);
    }
    return cudaGetLastError();
}

cudaError_t launch_morton(const BatchBuffers& b, cudaStream_t s) {
    if (b.radix_bits == 4)
        return launch_step(k_morton<4>, b.ntiles, kMortonThreads, 0, s, b.sims, b.tiles, b.minmax,
                           b.keys_a, b.hist, (uint32_t*)b.agg_region, b.simout);
    return launch_step(k_morton<8>, b.ntiles, kMortonThreads, 0, s, b.sims, b.tiles, b.minmax,
                       b.keys_a, b.hist, (uint32_t*)b.agg_region, b.simout);
}

// Passes alternate a -> b -> a ...; an even pass count leaves the sorted keys
// in keys_a, and the last pass also gathers the sorted bodies (with their indices).
// Streaming multiprocessors of the current device (cached per device).
static int sm_count() {
    static int cached[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    if (!cached[dev]) {
        int n = 0;
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        cached[dev] = n > 0 ? n : 148;
    }
    return cached[dev];
}

template <int BITS, int PASS>
static cudaError_t radix_passes(const BatchBuffers& b, cudaStream_t s) {
    constexpr int kPasses = 32 / BITS;
    const size_t fstride = (size_t)b.ntiles << BITS;
    const bool even = (PASS % 2) == 0;
    const uint32_t* kin = even ? b.keys_a : b.keys_b;
    const uint32_t* vin = even ? b.vals_a : b.vals_b;
    uint32_t* kout = even ? b.keys_b : b.keys_a;
    uint32_t* vout = even ? b.vals_b : b.vals_a;
    // more than two waves of tiles at two per SM: three per SM instead
    const bool many = b.ntiles > 2u * 2u * (uint32_t)sm_count();
    const cudaError_t e =
        many ? launch_step(k_radix_pass<BITS, PASS, PASS == kPasses - 1, 3>, b.ntiles,
                           kSortThreads, 0, s, b.sims, b.tiles, b.counters + PASS, b.hist,
                           b.sort_flags + PASS * fstride, (uint32_t*)b.agg_region, kin, PASS == 0 ? nullptr : vin, kout,
                           vout, b.sbody, b.err)
             : launch_step(k_radix_pass<BITS, PASS, PASS == kPasses - 1, 2>, b.ntiles,
                           kSortThreads, 0, s, b.sims, b.tiles, b.counters + PASS, b.hist,
                           b.sort_flags + PASS * fstride, (uint32_t*)b.agg_region, kin, PASS == 0 ? nullptr : vin, kout,
                           vout, b.sbody, b.err);
    if (e != cudaSuccess) return e;
    if constexpr (PASS + 1 < kPasses) return radix_passes<BITS, PASS + 1>(b, s);
    return cudaSuccess;
}

cudaError_t launch_radix(const BatchBuffers& b, cudaStream_t s) {
    return b.radix_bits == 4 ? radix_passes<4, 0>(b, s) : radix_passes<8, 0>(b, s);
}

// Lays the plan out in its region, which holds 24 bytes per cell (at least 24 a
// body, 768 in all): per block a cut and, by range, up to 256 bytes of inner list,
// per range the count and the outer list's 20 KB of cells.
static AggPlan agg_plan(const BatchBuffers& b) {
    AggPlan p;
    p.blocks = (b.npos + kAggPositions - 1) / kAggPositions;
    p.range = agg_range(p.blocks);
    p.ranges = (p.blocks + p.range - 1) / p.range;
    p.outer_n = b.counters + 16;
    char* at = (char*)b.agg_region;
    auto take = [&](size_t bytes) {
        char* q = at;
        at += (bytes + 15) & ~(size_t)15;
        return q;
    };
    p.inner_n = (uint32_t*)take(4ull * p.ranges);
    p.cuts = (uint32_t*)take(4ull * (p.blocks + 1));
    const size_t outer = p.ranges > 1 ? (size_t)kMortonDepth * p.ranges : 0;
    p.outer = (uint4*)take(sizeof(uint4) * outer);
    p.outer_cells = (SpanCell*)take(sizeof(SpanCell) * outer);
    p.inner = (uint4*)at;  // the last range's list is as long as its cuts allow
    return p;
}

// Blocks that a cluster of the largest k_sort_small may have here: 16, or the
// portable 8 where no part of the GPU holds 16 of them at once (a slice of it).
static uint32_t sort_cluster_limit() {
    static uint32_t cached[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 8;
    if (!cached[dev]) {
        auto kernel = k_sort_small<12, true, true, false>;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = kSmallBlocks;
        cfg.blockDim = kSmallThreads;
        cfg.dynamicSmemBytes = sizeof(SmallSort<12>);
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = kSmallBlocks;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int clusters = 0;
        const bool fits =
            cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(SmallSort<12>)) == cudaSuccess &&
            cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
                cudaSuccess &&
            cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) == cudaSuccess && clusters > 0;
        if (!fits) cudaGetLastError();
        cached[dev] = fits ? kSmallBlocks : 8u;
    }
    return cached[dev];
}

// The form of k_sort_small that a batch gets: 2^log positions a block, `cluster`
// blocks a simulation; log 0 for separate Morton, radix and scan launches (also
// where the caller asked for 4-bit digits).  The fewest positions a block while
// the batch has at most 64 blocks, since a block's time grows with them and the
// chip has room: 8 simulations of 8,192 bodies 109, 114 and 125 us a step at 1,024,
// 2,048 and 4,096; with 16 of them it is 149, 148 and 159, and 16 of 16,384 253, 243
// and 243.  Not in clusters of two: 71 us against 70 in one block at 2,048 bodies.
// With more than 64 blocks of 4,096 the chip is full, and clusters of 8 and 16,
// partly idle where simulations differ, lose to the tiles of k_radix_pass: 16 of
// 32,768 bodies 435 us against 421, 8 of 65,536 459 against 442, 96 of 2^10 to 2^16
// 1,133 against 1,033; of at most 4 they do not (32 of 16,384 393 against 405).
// No clusters where another stream keeps the GPU busy (b.clusters): one starts
// when enough neighbouring multiprocessors have room at the same time, and twelve
// requests' boundary solves beside the rounds of a server took 39 ms against 35.
struct SortForm {
    uint32_t log, cluster;
};
static SortForm sort_form(const BatchBuffers& b) {
    constexpr uint32_t kRoom = 64;
    if (b.radix_bits != 8 || b.max_bodies > kSmallSort) return {0, 0};
    for (uint32_t log = 10; log <= 12; ++log) {
        uint32_t cluster = 1;
        while (cluster << log < b.max_bodies) cluster *= 2;
        const uint64_t blocks = (uint64_t)cluster * b.nsims;
        if (cluster > 1 && !b.clusters) continue;
        if (cluster == 1 || (cluster > 2 && blocks <= kRoom && cluster <= sort_cluster_limit()) ||
            (log == 12 && cluster <= 4))
            return {log, cluster};
    }
    return {0, 0};
}

bool small_sort(const BatchBuffers& b) { return sort_form(b).log != 0; }

template <int LOG, bool SCAN, bool CLUSTER, bool TIMED = false>
static cudaError_t sort_small(const BatchBuffers& b, int mode, uint32_t cluster, cudaStream_t s) {
    auto kernel = k_sort_small<LOG, SCAN, CLUSTER, TIMED>;
    constexpr int bytes = (int)sizeof(SmallSort<LOG>);
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess && cluster > 8)
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    return launch_clusters(kernel, cluster, b.nsims * cluster, kSmallThreads, bytes, s, b.sims,
                           mode, b.npos, b.keys_a, b.sbody, b.base, agg_plan(b), b.simout,
                           b.err + kStageCycles);
}

template <int LOG>
static cudaError_t sort_small(const BatchBuffers& b, int mode, bool timed, uint32_t cluster,
                              cudaStream_t s) {
    if (b.nsims == 1 && timed)
        return cluster == 1 ? sort_small<LOG, true, false, true>(b, mode, cluster, s)
                            : sort_small<LOG, true, true, true>(b, mode, cluster, s);
    if (b.nsims == 1)
        return cluster == 1 ? sort_small<LOG, true, false>(b, mode, cluster, s)
                            : sort_small<LOG, true, true>(b, mode, cluster, s);
    return cluster == 1 ? sort_small<LOG, false, false>(b, mode, cluster, s)
                        : sort_small<LOG, false, true>(b, mode, cluster, s);
}

cudaError_t launch_sort_small(const BatchBuffers& b, int mode, bool timed, cudaStream_t s) {
    const SortForm f = sort_form(b);
    return f.log == 10   ? sort_small<10>(b, mode, timed, f.cluster, s)
           : f.log == 11 ? sort_small<11>(b, mode, timed, f.cluster, s)
                         : sort_small<12>(b, mode, timed, f.cluster, s);
}

cudaError_t launch_count_scan(const BatchBuffers& b, cudaStream_t s) {
    return launch_step(k_count_scan, b.nscan_tiles, kScanThreads, 0, s, b.sims, b.chunk_sim,
                       b.npos, b.keys_a, b.base, agg_plan(b), b.counters + 8, b.scan_flags, b.err);
}

cudaError_t launch_aggregate(const BatchBuffers& b, cudaStream_t s) {
    const AggArgs a{b.sims,          b.simout, b.chunk_sim, b.sbody,  b.keys_a,
                    b.cell_capacity, b.base,   b.cell_u,    b.cell_d, b.groups, b.nsims};
    const AggPlan plan = agg_plan(b);
    cudaError_t e = launch_step(k_aggregate, plan.blocks, kAggThreads, 0, s, a, plan, b.err);
    if (e == cudaSuccess && plan.blocks > 1) {
        const uint32_t outer =
            plan.ranges > 1 ? (kMortonDepth * plan.ranges + kSpanThreads - 1) / kSpanThreads : 0;
        e = launch_step(k_aggregate_inner, plan.ranges + outer, kSpanThreads, 0, s, a, plan);
    }
    if (e == cudaSuccess && plan.ranges > 1)
        e = launch_step(k_aggregate_outer, 1, kSpanThreads, 0, s, a, plan);
    return e;
}

cudaError_t launch_wait_probe(uint32_t* words, uint32_t* err, long long limit, uint32_t* out,
                              cudaStream_t s) {
    k_wait_probe<<<2, kRadixDigits, 0, s>>>(words, err, limit > 0 ? limit : kSpinCycles, out);
    return cudaGetLastError();
}

cudaError_t launch_refresh_mac(const BatchBuffers& b, uint32_t sim, cudaStream_t s) {
    k_refresh_mac<<<(b.cell_capacity + 255) / 256, 256, 0, s>>>(
        b.sims, b.simout, sim, b.base, b.keys_a, b.cell_capacity,
        b.cell_d, b.cell_u, b.groups);
    return cudaGetLastError();
}

template <int WARPS, bool NORMAL>
static cudaError_t traverse_launch(const BatchBuffers& b, bool compensated, bool potential,
                                   bool stats, cudaStream_t s) {
    // The compensated form keeps a residual per list entry; with it 8 warps'
    // static shared memory would pass 48 KB, so it runs at most 4 warps per
    // block (each warp does the same work at any block size).
    constexpr int CW = WARPS > 4 ? 4 : WARPS;
#define GBH_TRAVERSE(C, P, S)                                                                   \
    return launch_step(k_traverse<C, P, S, (C ? CW : WARPS), NORMAL>,                           \
                       (b.nchunks + (C ? CW : WARPS) - 1) / (C ? CW : WARPS),                   \
                       (C ? CW : WARPS) * 32, 0, s, b.sims, b.simout, b.chunk_sim, b.nchunks,  \
                       b.sbody, b.groups, b.cell_d, b.cell_capacity, b.force_stats, b.err)
    if (stats) {
        if (compensated) {
            if (potential) GBH_TRAVERSE(true, true, true);
            GBH_TRAVERSE(true, false, true);
        }
        if (potential) GBH_TRAVERSE(false, true, true);
        GBH_TRAVERSE(false, false, true);
    }
    if (compensated) {
        if (potential) GBH_TRAVERSE(true, true, false);
        GBH_TRAVERSE(true, false, false);
    }
    if (potential) GBH_TRAVERSE(false, true, false);
    GBH_TRAVERSE(false, false, false);
#undef GBH_TRAVERSE
}

template <bool NORMAL>
static cudaError_t traverse_warps(const BatchBuffers& b, bool compensated, bool potential,
                                  bool stats, cudaStream_t s) {
    if (b.trav_warps == 2) return traverse_launch<2, NORMAL>(b, compensated, potential, stats, s);
    if (b.trav_warps == 4) return traverse_launch<4, NORMAL>(b, compensated, potential, stats, s);
    return traverse_launch<kTravWarps, NORMAL>(b, compensated, potential, stats, s);
}

// The general form where the softening's square is subnormal (or zero) in some
// simulation of the batch.
static cudaError_t traverse_form(const BatchBuffers& b, bool compensated, bool potential,
                                 bool stats, cudaStream_t s) {
    return b.normal_eps2 ? traverse_warps<true>(b, compensated, potential, stats, s)
                         : traverse_warps<false>(b, compensated, potential, stats, s);
}

cudaError_t launch_traverse(const BatchBuffers& b, bool compensated, bool plain, bool potential,
                            bool stats, cudaStream_t s) {
    cudaError_t e = cudaSuccess;
    if (compensated) e = traverse_form(b, true, potential, stats, s);
    if (e == cudaSuccess && plain) e = traverse_form(b, false, potential, stats, s);
    return e;
}

cudaError_t launch_export(const BatchBuffers& b, uint32_t sim, GpuEntry* entries, GpuBody* bodies,
                          GpuCell* cells, cudaStream_t s) {
    if (cells)
        k_export_cells<<<(b.cell_capacity + 255) / 256, 256, 0, s>>>(
            b.sims, b.simout, sim, b.keys_a, b.base, b.cell_u, b.cell_d,
            cells);
    if (entries || bodies)
        k_export_entries<<<(b.npos + 255) / 256, 256, 0, s>>>(b.sims, sim, b.keys_a, b.sbody,
                                                             entries, bodies);
    return cudaGetLastError();
}

cudaError_t launch_traverse_packed(const BhSettings* settings, const GpuBody* bodies,
                                   const GpuEntry* entries, const GpuCell* cells, uint32_t n,
                                   uint32_t ncells, float4* accel, uint32_t* err,
                                   cudaStream_t s) {
    // err[1]: set when the entries and bodies disagree (the walk then goes
    // cell by cell)
    k_check_packed<<<(n + 255) / 256, 256, 0, s>>>(bodies, entries, n, err + 1);
    const uint32_t warps = (n + 31) / 32;
    k_traverse_packed<<<(warps + kPkWarps - 1) / kPkWarps, kPkWarps * 32, 0, s>>>(
        settings, bodies, entries, cells, n, ncells, accel, err, err + 1);
    return cudaGetLastError();
}

uint32_t conservation_blocks(uint32_t n) {
    uint32_t blocks = (n + kConsThreads - 1) / kConsThreads;
    return blocks < 592u ? (blocks ? blocks : 1u) : 592u;
}

cudaError_t launch_conservation(const GpuEvolveState* state, const float* potential, uint32_t n,
                                double* partials, uint32_t nblocks, double* out,
                                cudaStream_t s) {
    k_conservation_partial<<<nblocks, kConsThreads, 0, s>>>(state, potential, n, partials);
    k_conservation_final<<<1, 32 * kConsTerms, 0, s>>>(partials, nblocks, out);
    return cudaGetLastError();
}


// ============================================================ checks ====

// The readback checks of nbody_gpu.rs:1043-1053 (states) and 1097-1101
// (accelerations), evaluated on the device copy of the records.
template <int KIND>
__global__ void __launch_bounds__(256) k_check_records(const float4* __restrict__ rec, uint32_t n,
                                                       uint32_t* first_bad) {
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        bool ok;
        if (KIND == 0) {
            const float4 pm = rec[2ull * i];
            const float4 v = rec[2ull * i + 1];
            ok = isfinite(pm.x) && isfinite(pm.y) && isfinite(v.x) && isfinite(v.y) &&
                 isfinite(pm.z) && pm.z > 0.f;
        } else {
            const float4 a = rec[i];
            ok = isfinite(a.x) && isfinite(a.y);
        }
        if (!ok) atomicMin(first_bad, i);
    }
}

cudaError_t launch_check_records(const void* records, int kind, uint32_t n, uint32_t* first_bad,
                                 cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const uint64_t want = (n + 255ull) / 256ull;
    const uint32_t blocks = (uint32_t)(want < 148ull * 16ull ? want : 148ull * 16ull);
    if (kind == 0)
        k_check_records<0><<<blocks, 256, 0, s>>>(static_cast<const float4*>(records), n, first_bad);
    else
        k_check_records<1><<<blocks, 256, 0, s>>>(static_cast<const float4*>(records), n, first_bad);
    return cudaGetLastError();
}

}  // namespace gbh
