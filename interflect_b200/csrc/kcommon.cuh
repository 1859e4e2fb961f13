// Shared kernel prologue: make the scene program visible to the CTA, and the
// persistent ray-queue machinery the tracing kernels share.
#pragma once

#include "device.cuh"
#include "kernels.h"
#include "rowspan.h"

namespace ifx {

static constexpr int kWarp = 32;
static constexpr unsigned kFull = 0xffffffffu;

// Dynamic shared memory of a tracing CTA: the staged blob (when it fits)
// followed by the threads' BVH stacks.
static inline size_t blob_smem(const BlobRef& b, int block) {
    size_t s = b.staged ? (size_t)align16(b.stage_bytes) : 0;
    return s + (size_t)b.stack_depth * (size_t)block * 8u;  // node index + box distance
}

// Stages the blob's geometry prefix into dynamic shared memory (one bulk
// copy) or, for large scenes, reads it in place, and points the view at this
// thread's stack. All threads of the CTA must call this before any of them
// exits. Returns false if staging timed out.
__device__ __forceinline__ bool scene_prologue(const BlobRef& blob, uint8_t* dsmem, uint64_t* mbar,
                                               uint32_t* status, SceneView& sv) {
    sv = make_view(blob.ptr);
    sv.status = status;
    sv.og = blob.og;
    uint32_t used = 0;
    if (blob.staged) {
        if (!stage_scene(blob.ptr, blob.stage_bytes, dsmem, mbar, status, blob.wait_polls)) return false;
        const SceneView s = make_view(dsmem);
        sv.objs = s.objs;
        sv.prims = s.prims;
        sv.nodes = s.nodes;
        sv.fast = s.fast;
        used = align16(blob.stage_bytes);
    }
    uint32_t* stk = reinterpret_cast<uint32_t*>(dsmem + used);
    sv.stk = stk + threadIdx.x;
    sv.stkd = reinterpret_cast<float*>(stk + (size_t)blob.stack_depth * blockDim.x) + threadIdx.x;
    sv.stk_stride = (int)blockDim.x;
    sv.stk_depth = blob.stack_depth;
    return true;
}

#define IFX_SCENE_PROLOGUE(blob, status, sv)                                  \
    extern __shared__ __align__(128) uint8_t ifx_dsmem[];                     \
    __shared__ __align__(8) uint64_t ifx_mbar;                                \
    SceneView sv;                                                             \
    if (!scene_prologue(blob, ifx_dsmem, &ifx_mbar, status, sv)) return;

// Bounded grid barrier over the CTAs of one cooperative launch (every CTA is
// resident, so all of them arrive unless one has left after an error).
// Returns false, with kStatusBarrier set in *status, when the other CTAs did
// not arrive within `polls` polls; the caller then leaves the kernel. The
// barrier's count must be zero at launch.
static constexpr uint32_t kStatusBarrier = 1u << 4;
__device__ __forceinline__ bool grid_barrier(MsBarrier* b, uint32_t* status, uint32_t polls) {
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        ok = 1;
        volatile uint32_t* vgen = &b->gen;
        const uint32_t g = *vgen;
        __threadfence();
        if (atomicAdd(&b->count, 1u) == gridDim.x - 1) {
            atomicExch(&b->count, 0u);
            __threadfence();
            atomicAdd(&b->gen, 1u);
        } else {
            uint32_t n = 0;
            while (*vgen == g) {
                if (++n > polls) {
                    atomicOr(status, kStatusBarrier);
                    ok = 0;
                    break;
                }
                __nanosleep(128);
            }
        }
        __threadfence();
    }
    __syncthreads();
    return ok != 0;
}

// Number of CTAs for a grid-stride kernel: enough to fill every SM several
// times over, never more than the work needs.
static inline int sm_count() {
    static int cached[64] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    if (!cached[dev]) {
        int sms = 148;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cached[dev] = sms;
    }
    return cached[dev];
}

// Calls f with the counter policy that a tracing kernel takes for the scene:
// the counting kernels, or by its tree and by whether it has an object grid.
template <class C>
struct Policy {
    using type = C;
};
template <class F>
static inline void with_policy(const BlobRef& b, bool counts, F&& f) {
    if (counts) f(Policy<Counts>{});
    else if (b.og.mode == kOgOff && b.tree3) f(Policy<NoGrid3>{});
    else if (b.og.mode == kOgOff) f(Policy<NoGrid>{});
    else if (b.tree3) f(Policy<NoCount3>{});
    else f(Policy<NoCount>{});
}
// The policies of scenes without a grid, or the others.
template <class F>
static inline void for_each_policy(bool no_grid, F&& f) {
    if (no_grid) {
        f(Policy<NoGrid3>{});
        f(Policy<NoGrid>{});
    } else {
        f(Policy<Counts>{});
        f(Policy<NoCount3>{});
        f(Policy<NoCount>{});
    }
}

static inline unsigned grid_for(unsigned long long items, int block, int per_sm_ctas = 8) {
    unsigned long long need = (items + (unsigned long long)block - 1) / (unsigned long long)block;
    unsigned long long cap = (unsigned long long)sm_count() * (unsigned long long)per_sm_ctas;
    if (need < 1) need = 1;
    return (unsigned)(need < cap ? need : cap);
}

// Persistent kernels: one wave of CTAs, as many as are co-resident. Few items
// are spread thinly (WarpQueue then leaves lanes of every warp empty) until
// there are kSpreadCtas per SM: a warp issues at most every fourth cycle or so
// along a ray's dependent chain, so a scheduler needs about five warps to
// stay busy, and a warp of fewer rays takes fewer divergent turns per step. Not
// so without a BVH, where all rays of a warp evaluate the same objects and more
// warps do the same work again (40 objects, 97 x 61: 2.33 -> 2.63 ms spread).
static constexpr unsigned kSpreadCtas = 5;
template <class K>
static inline unsigned persistent_grid(K kernel, int block, size_t smem, unsigned long long items, const BlobRef& blob) {
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, smem);
    if (per_sm < 1) per_sm = 1;
    unsigned long long cap = (unsigned long long)sm_count() * (unsigned long long)per_sm;
    unsigned long long need = (items + (unsigned long long)block - 1) / (unsigned long long)block;
    const unsigned long long thin = (items * 32ull + (unsigned long long)block - 1) / (unsigned long long)block;
    const unsigned long long spread = blob.linear ? 0ull : (unsigned long long)sm_count() * kSpreadCtas;
    need = need > spread ? need : (thin < spread ? thin : spread);
    if (need < 1) need = 1;
    return (unsigned)(need < cap ? need : cap);
}

// Warp-level work distribution for persistent ray kernels. Every lane holds
// at most one item (a ray); lanes whose ray finished are refilled from the
// warp's private range of item indices, which is replenished in chunks of
// kChunk indices from a global cursor with one atomic per chunk. Which lane
// or warp traces an item never affects its result: each item's output is
// written to a slot fixed by its index.
// Lanes wait until kRefill of 32 are idle (or as large a share of those in
// use): starting a ray costs about a third of a step (loads, divisions and
// roots), and all lanes pay for it however few start. At 1, 4, 8, 12, 16: the
// 512-object scene's visibility 17.8, 16.5, 16.6, 17.1, 17.7 ms, the product
// scene's shadow rays 1.01, 0.94, 0.91, 0.89, 0.90 ms, its camera rays 0.72,
// 0.72, 0.74, 0.83, 0.87 ms. Without a grid a step is dearer and an idle lane
// costs more than a start: those kernels refill at one.
static constexpr uint32_t kRefill = 8;
template <class C>
struct WarpQueue {
    uint32_t cur, end;  // warp-uniform private range [cur, end)
    uint32_t kChunk;    // items taken per atomic: about 1/8 of a fair share per warp, 32..256, or
                        // the whole share where it is less than a warp
    uint32_t lanes;     // lanes that take items: all, or a fair share where there are few items
    bool drained;

    __device__ __forceinline__ explicit WarpQueue(unsigned long long total) : cur(0), end(0), drained(false) {
        const unsigned long long warps = (unsigned long long)gridDim.x * blockDim.x / 32u;
        unsigned long long c = total / (warps * 8ull + 1ull);
        c = c < 32ull ? 32ull : (c > 256ull ? 256ull : c);
        const unsigned long long share = (total + warps - 1ull) / warps;
        // At least one, of an empty queue too: some lane has to find it drained.
        lanes = share < 1ull ? 1u : (share < 32ull ? (uint32_t)share : 32u);
        kChunk = lanes < 32u ? lanes : (uint32_t)(c & ~31ull);
    }

    // Returns the item for this lane (or ~0u) when it is idle; `idle` says
    // whether this lane needs an item. Must be called by all 32 lanes.
    __device__ __forceinline__ uint32_t refill(bool idle, unsigned long long total, unsigned long long* cursor) {
        const int lane = threadIdx.x & 31;
        idle = idle && (uint32_t)lane < lanes;
        unsigned need = __ballot_sync(kFull, idle);
        uint32_t item = ~0u;
        if ((uint32_t)__popc(need) < (C::kGrid ? kRefill : 1u) * lanes / 32u || !need) return item;
        if (cur >= end && !drained) {
            unsigned long long base = 0;
            if (lane == 0) base = atomicAdd(cursor, (unsigned long long)kChunk);
            base = __shfl_sync(kFull, base, 0);
            if (base >= total) {
                drained = true;
            } else {
                cur = (uint32_t)base;
                end = (uint32_t)(base + kChunk < total ? base + kChunk : total);
            }
        }
        if (cur < end) {
            uint32_t avail = end - cur;
            uint32_t rank = __popc(need & ((1u << lane) - 1u));
            if (idle && rank < avail) item = cur + rank;
            uint32_t k = __popc(need);
            cur += k < avail ? k : avail;
        }
        return item;
    }
    __device__ __forceinline__ bool empty() const { return drained && cur >= end; }
};

// Programmatic dependent launch between the kernels of a bounce, forward or
// adjoint: a kernel starts
// by waiting until the previous kernel in its stream has completed and its
// writes are visible (pdl_wait), and once its main loop is done it lets the
// next kernel be scheduled (pdl_trigger), whose CTAs then wait in their own
// pdl_wait. Both are no-ops in a launch without the programmatic attribute.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// A bounce kernel launched with the programmatic-serialization attribute:
// the stream (or the captured graph's edge) lets it start once the previous
// kernel has triggered, and pdl_wait orders its work after that kernel.
template <typename... K, typename... A>
static inline void launch_pdl(void (*kernel)(K...), unsigned grid, unsigned block, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, args...);
}

// ------------------------------------------------------ Jacobi bounces ----
// solve.rs:93-101: whether the solve has stopped before bounce `it`. Every
// thread of a bounce's first phase decides the same, whether or not it sees
// solve_note's writes. A kernel that runs through several bounces passes a
// volatile block: what L1 holds of it may be a bounce old. One that is launched
// for its bounce passes a plain one, whose words an SM's warps find in L1:
// volatile, every warp of thousands of CTAs went to one place in L2 (2,500
// clusters: 10.1 -> 8.4 us a bounce's means, 7.6 -> 3.7 us past convergence).
template <class Ctl>
__device__ __forceinline__ bool solve_stopped(const Ctl& c, uint32_t it, int no_exit) {
    const uint32_t done = c.done, res = c.res[(it - 1) & 1];
    return done || (!no_exit && it > 0 && __uint_as_float(res) < 1e-4f);
}
// One thread's part before bounce `it`: the statistics of the bounces so far.
__device__ __forceinline__ void solve_note(SolveCtl& c, uint32_t it, bool stop) {
    if (c.done) return;
    if (it > 0) {
        c.iterations = it;
        c.last_residual = c.res[(it - 1) & 1];
    }
    if (stop) c.done = 1;
    else c.res[it & 1] = 0;
}

// solve.rs:76-102: the sum of a row's links [k, e) in CSR order (the
// reference's sum). Each turn issues the index and weight loads of 8 links as
// two 128-bit loads each, then the 8 cluster gathers, before the first add, so
// a thread keeps 12 loads in flight; the products crad[idx] * w and their
// left-to-right sum round exactly as the scalar loop does. `vec` is 0 when
// idx or w is not 16-byte aligned (caller-provided arrays), which keeps every
// load scalar.
__device__ __forceinline__ V jacobi_row(const float4* crad, const uint32_t* __restrict__ idx,
                                        const float* __restrict__ w, uint32_t k, uint32_t e, int vec) {
    V irr{0.0f, 0.0f, 0.0f};
    if (vec) {
        for (; k < e && (k & 3u); ++k) irr = irr + mk4(crad[__ldg(&idx[k])]) * __ldg(&w[k]);
        for (; span_full(k, e); k += kSpan) {
            const uint4 i0 = __ldg(reinterpret_cast<const uint4*>(idx + k));
            const uint4 i1 = __ldg(reinterpret_cast<const uint4*>(idx + k + 4));
            const float4 w0 = __ldg(reinterpret_cast<const float4*>(w + k));
            const float4 w1 = __ldg(reinterpret_cast<const float4*>(w + k + 4));
            const float4 c0 = crad[i0.x], c1 = crad[i0.y], c2 = crad[i0.z], c3 = crad[i0.w], c4 = crad[i1.x],
                         c5 = crad[i1.y], c6 = crad[i1.z], c7 = crad[i1.w];
            irr = irr + mk4(c0) * w0.x;
            irr = irr + mk4(c1) * w0.y;
            irr = irr + mk4(c2) * w0.z;
            irr = irr + mk4(c3) * w0.w;
            irr = irr + mk4(c4) * w1.x;
            irr = irr + mk4(c5) * w1.y;
            irr = irr + mk4(c6) * w1.z;
            irr = irr + mk4(c7) * w1.w;
        }
    }
    for (; k < e; ++k) irr = irr + mk4(crad[__ldg(&idx[k])]) * __ldg(&w[k]);
    return irr;
}

// solve.rs:76-102 over the sliced-ELL copy: one thread per sorted position
// (its warp is its slice), the row's links read 4 at a time as 128-bit loads
// from the interleaved layout (a warp's loads are one contiguous 512-byte
// block) and added in CSR order, exactly as k_jacobi; a lane stops at its own
// row's length, so padding is never read. Outputs go to the original row.
// The next 8 links' indices and weights are loaded while the current ones are
// gathered and added: with few rows the kernel is one such chain per row.
__device__ __forceinline__ V sell_row(const SellMatrix& m, const float4* crad, uint32_t sp, uint32_t len) {
    const uint4* ip = reinterpret_cast<const uint4*>(m.idx + m.slice_off[sp >> 5] + (sp & 31u) * 4u);
    const float4* wp = reinterpret_cast<const float4*>(m.w + m.slice_off[sp >> 5] + (sp & 31u) * 4u);
    V irr{0.0f, 0.0f, 0.0f};
    if (len == 0) return irr;
    // Entries [0, 4 * ceil(len / 4)) of the row exist (padding included).
    uint4 i0 = __ldg(ip), i1 = len > 4u ? __ldg(ip + 32) : i0;
    float4 w0 = __ldg(wp), w1 = len > 4u ? __ldg(wp + 32) : w0;
    for (uint32_t j = 0;; j += 8) {
        const uint32_t left = len - j;
        const uint4 a0 = i0, a1 = i1;
        const float4 b0 = w0, b1 = w1;
        ip += 64;
        wp += 64;
        if (left > 8u) {
            i0 = __ldg(ip);
            w0 = __ldg(wp);
        }
        if (left > 12u) {
            i1 = __ldg(ip + 32);
            w1 = __ldg(wp + 32);
        }
        if (left >= 8u) {
            const float4 c0 = crad[a0.x], c1 = crad[a0.y], c2 = crad[a0.z], c3 = crad[a0.w], c4 = crad[a1.x],
                         c5 = crad[a1.y], c6 = crad[a1.z], c7 = crad[a1.w];
            irr = irr + mk4(c0) * b0.x;
            irr = irr + mk4(c1) * b0.y;
            irr = irr + mk4(c2) * b0.z;
            irr = irr + mk4(c3) * b0.w;
            irr = irr + mk4(c4) * b1.x;
            irr = irr + mk4(c5) * b1.y;
            irr = irr + mk4(c6) * b1.z;
            irr = irr + mk4(c7) * b1.w;
            if (left == 8u) return irr;
        } else {
            const uint32_t ia[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
            const float wa[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
            for (uint32_t t = 0; t < 7u; ++t)
                if (t < left) irr = irr + mk4(crad[ia[t]]) * wa[t];
            return irr;
        }
    }
}

}  // namespace ifx
