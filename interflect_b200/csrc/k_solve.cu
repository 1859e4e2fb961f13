// Direct light on surfels (solve.rs:27-39; for many (surfel, light) slots
// the light stage uses launch_light_slots in k_shade.cu instead) and the
// Jacobi bounce solve (solve.rs:47-108). The bounce loop runs without host round trips: every
// bounce kernel first reads a device-side control block, so the host enqueues
// many bounces at once and the ones after convergence return immediately. A
// bounce is two launches, the cluster means and the rows: the stop test is
// part of the next bounce's first kernel (SolveCtl).
#include "kcommon.cuh"

namespace ifx {

__device__ __forceinline__ void block_add_u64(unsigned long long v, unsigned long long* out) {
    for (int o = 16; o >= 1; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(out, v);
}

// solve.rs:27-39
template <class C>
__global__ void __launch_bounds__(128) k_light_surfels(BlobRef blob, SurfelArrays s, uint32_t n,
                                                        unsigned long long* evals, uint32_t* status,
                                                        unsigned long long* counts, float* terms) {
    IFX_SCENE_PROLOGUE(blob, status, sv);
    C cnt;
    const uint32_t stride = gridDim.x * blockDim.x;
    const uint32_t limit = (n + stride - 1) / stride * stride;  // keep whole warps for the reduction
    const int nl = sv.n_lights + sv.n_slights;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < limit; i += stride) {
        unsigned long long e = 0;
        if (i < n) {
            uint32_t steps = 0;
            V c = direct_diffuse(sv, mk4(s.p[i]), mk4(s.n[i]), mk4(s.albedo[i]), steps, cnt,
                                 terms ? terms + (size_t)i * nl : nullptr);
            s.direct[i] = f4(c, 0.0f);
            s.rad[i] = f4(c, 0.0f);
            s.irr[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            e = steps;
        }
        block_add_u64(e, evals);
    }
    if constexpr (sizeof(C) > 1) cnt.flush(counts);
}

// solve.rs:61-73: cluster radiosity as the area-weighted mean of its
// members' radiosity, summed sequentially in member order, by one CTA: the
// threads gather members' rad * area (each product exact per element) into
// shared memory chunk by chunk, double-buffered, and thread 0 adds them in
// member order.
template <int kBlock>
__device__ __forceinline__ void cluster_mean(const float4* rad, const float4* sp, const float4* cp,
                                             const uint2* crange, const uint32_t* members, uint32_t c,
                                             float4* cluster_rad, float4 (*buf)[kBlock]) {
    const uint2 r = crange[c];
    const uint32_t len = r.y - r.x;
    const uint32_t chunks = (len + kBlock - 1) / kBlock;
    auto load = [&](uint32_t ch, int b) {
        uint32_t k = r.x + ch * kBlock + threadIdx.x;
        if (k < r.y) {
            uint32_t m = __ldg(&members[k]);
            float4 v = __ldg(&rad[m]);
            float a = __ldg(&sp[m].w);
            buf[b][threadIdx.x] = make_float4(v.x * a, v.y * a, v.z * a, 0.0f);
        }
    };
    if (chunks) load(0, 0);
    __syncthreads();
    V acc{0.0f, 0.0f, 0.0f};
    for (uint32_t ch = 0; ch < chunks; ++ch) {
        const int b = ch & 1;
        if (threadIdx.x == 0) {
            const uint32_t cnt = min((uint32_t)kBlock, len - ch * kBlock);
            // Unrolled so that the shared-memory loads run ahead of the
            // chain of additions (which stays in member order).
            uint32_t k = 0;
            for (; k + 8 <= cnt; k += 8) {
                float4 v[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = buf[b][k + j];
#pragma unroll
                for (int j = 0; j < 8; ++j) acc = acc + V{v[j].x, v[j].y, v[j].z};
            }
            for (; k < cnt; ++k) {
                float4 v = buf[b][k];
                acc = acc + V{v.x, v.y, v.z};
            }
            if (ch + 1 < chunks) load(ch + 1, b ^ 1);
        } else if (ch + 1 < chunks) {
            load(ch + 1, b ^ 1);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) cluster_rad[c] = f4(acc / fmaxf(__ldg(&cp[c].w), 1e-12f), 0.0f);
    __syncthreads();
}

static constexpr int kAggBlock = 128;
__global__ void __launch_bounds__(kAggBlock) k_cluster_agg(const float4* rad, const float4* sp, const float4* cp,
                                                            const uint2* crange, const uint32_t* members,
                                                            uint32_t nc, float4* cluster_rad, SolveCtl* ctl,
                                                            uint32_t it, int no_exit) {
    pdl_wait();
    const bool stop = solve_stopped(*ctl, it, no_exit);
    if (blockIdx.x == 0 && threadIdx.x == 0) solve_note(*ctl, it, stop);
    if (stop) return;
    __shared__ float4 buf[2][kAggBlock];
    for (uint32_t c = blockIdx.x; c < nc; c += gridDim.x)
        cluster_mean<kAggBlock>(rad, sp, cp, crange, members, c, cluster_rad, buf);
    pdl_trigger();
}

// solve.rs:76-102, one row per thread. The bounce residual is the maximum
// change over rows, an order-free reduction kept as the bits of a non-negative
// f32 (NaN ignored, as the reference's f32::max fold does).
static constexpr int kJacBlock = 256;
__device__ __forceinline__ void note_residual(float dmax, SolveCtl* ctl, uint32_t it) {
    for (int o = 16; o >= 1; o >>= 1) dmax = fmaxf(dmax, __shfl_xor_sync(kFull, dmax, o));
    if ((threadIdx.x & 31) == 0 && dmax > 0.0f) atomicMax(&ctl->res[it & 1], __float_as_uint(dmax));
}

// The end of row i: irradiance, new radiosity, |change|.
__device__ __forceinline__ float row_update(const float4* direct, const float4* albedo, float4* irr_out, float4* rad,
                                            uint32_t i, V irr) {
    const V nr = mk4(__ldg(&direct[i])) + mk4(__ldg(&albedo[i])) * irr;
    const V diff = vabs(nr - mk4(rad[i]));
    irr_out[i] = f4(irr, 0.0f);
    rad[i] = f4(nr, 0.0f);
    const float d = fmaxf(diff.x, fmaxf(diff.y, diff.z));
    return isnan(d) ? 0.0f : d;
}

__global__ void __launch_bounds__(kJacBlock) k_jacobi(const float4* direct, const float4* albedo, float4* irr_out,
                                                       float4* rad, uint32_t n, const uint32_t* starts,
                                                       const uint32_t* idx, const float* w,
                                                       const float4* __restrict__ crad, SolveCtl* ctl, uint32_t it,
                                                       int vec) {
    pdl_wait();
    if (ctl->done) return;
    float dmax = 0.0f;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        dmax = fmaxf(dmax, row_update(direct, albedo, irr_out, rad, i,
                                      jacobi_row(crad, idx, w, starts[i], starts[i + 1], vec)));
    pdl_trigger();
    note_residual(dmax, ctl, it);
}

// Many rows: from here on they fill the GPU's warps.
static constexpr uint32_t kManyRows = 65536;
// The wide row walk: from so many rows on, and of so many links each in the
// mean. Fewer rows are one chain per link, which its masked ends lengthen, and
// the ends are a larger part of shorter rows. 8 bounces of scenes' transfers
// with 16-byte loads and wide, in us, by rows and mean links:
//            20,000     50,000     100,000    250,000      1,000,000
//    19   132, 158   158, 169   210, 221   422, 434   1,455, 1,530
//    35   166, 185   185, 194   244, 251   494, 505
//    57   211, 248   233, 238   303, 305   743, 708
//   109   310, 361   359, 344   567, 494   1,240, 1,137   3,830, 3,667
// and a Cornell box's 60,000 rows of 48 links 223, 231, of 119 links 345, 331.
static constexpr uint32_t kWideRows = 49152, kWideLinks = 64;
// Cluster radiosities gathered from shared memory: up to 4,096 clusters. Few
// rows take as long as the longest one's chain of gathers, each kernel with a
// cold L1: small CTAs spread them over the SMs, and up to 1,024 clusters a copy
// per CTA pays (20,000 rows, 793 clusters: 12 bounces 0.325 -> 0.258 ms; 50,000
// rows, 2,504 clusters, 40 KiB a copy: 0.44 -> 0.47 ms). It pays where a CTA
// gathers as many links as it copies clusters (8,000 rows of 5 links, 1,000
// clusters, 12 bounces: 89 us copied, 69 not).
static constexpr size_t kSharedRadMax = 64u * 1024u, kSharedRadSmall = 16u * 1024u;
static constexpr unsigned kFewRowsBlock = 128;

// Eight 32-bit words in one load; p is 32-byte aligned, its data constant.
__device__ __forceinline__ void load8(const void* p, uint32_t v[8]) {
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
        : "l"(p));
}

// A row's sum where idx and w are 32-byte aligned, as allocations are. The rows
// of a warp lie in 32 places, so each of its loads is 32 cache lines' worth of
// L1 cycles however little it takes: links come eight at a time in 256-bit
// loads of whole sectors, from the aligned place at or before the row's first
// link to the one at or after its last, those of the neighbouring rows masked.
// The stress scene's 1M rows and 109M links: 5.78 -> 4.76 ms for 14 bounces;
// as many rows and links drawn at random, 3.89 -> 3.39 ms. (With the cluster
// radiosities in shared memory the random matrix took 2.83 ms but the scene's
// 9.31: its rows differ in length and see the same clusters, which L1 serves
// in few lines. Tiles of 32 rows copied to shared memory first: 1.2 times the
// shared form on the random one.)
__device__ __forceinline__ V wide_row(const float4* __restrict__ crad, const uint32_t* idx, const float* w, uint32_t s,
                                      uint32_t e, uint32_t total) {
    V irr{0.0f, 0.0f, 0.0f};
    for (uint32_t k = s & ~(kSpan - 1u); k < e; k = span_next(k, e)) {
        uint32_t a[8], b[8];
        if (span_full(k, total)) {
            load8(idx + k, a);
            load8(w + k, b);
        } else {  // the last links of the matrix
#pragma unroll
            for (uint32_t t = 0; t < 8u; ++t) {
                a[t] = k + t < total ? __ldg(&idx[k + t]) : 0u;
                b[t] = k + t < total ? __float_as_uint(__ldg(&w[k + t])) : 0u;
            }
        }
        if (k >= s && span_full(k, e)) {
            float4 c[8];
#pragma unroll
            for (int t = 0; t < 8; ++t) c[t] = crad[a[t]];
#pragma unroll
            for (int t = 0; t < 8; ++t) irr = irr + mk4(c[t]) * __uint_as_float(b[t]);
        } else {
#pragma unroll
            for (uint32_t t = 0; t < 8u; ++t)
                if (k + t >= s && k + t < e) irr = irr + mk4(crad[a[t]]) * __uint_as_float(b[t]);
        }
    }
    return irr;
}

// The mean row length is known on the device alone, where the caller's arrays
// are: every thread decides alike by the number of links.
__global__ void __launch_bounds__(kJacBlock) k_jacobi_wide(const float4* direct, const float4* albedo,
                                                            float4* irr_out, float4* rad, uint32_t n,
                                                            const uint32_t* starts, const uint32_t* idx,
                                                            const float* w, const float4* __restrict__ crad,
                                                            SolveCtl* ctl, uint32_t it) {
    pdl_wait();
    if (ctl->done) return;
    const uint32_t total = starts[n];
    const bool wide = total >= (unsigned long long)n * kWideLinks;
    float dmax = 0.0f;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t s = starts[i], e = starts[i + 1];
        const V irr = wide ? wide_row(crad, idx, w, s, e, total) : jacobi_row(crad, idx, w, s, e, 1);
        dmax = fmaxf(dmax, row_update(direct, albedo, irr_out, rad, i, irr));
    }
    pdl_trigger();
    note_residual(dmax, ctl, it);
}

// solve.rs:93-101 after the last bounce that was launched.
__global__ void k_solve_end(SolveCtl* ctl, uint32_t it) {
    pdl_wait();
    const bool stop = solve_stopped(*ctl, it, 0);
    solve_note(*ctl, it, stop);
}

void launch_light_surfels(cudaStream_t st, BlobRef blob, SurfelArrays s, uint32_t n, unsigned long long* evals,
                          uint32_t* status, unsigned long long* counts, float* terms) {
    const unsigned g = grid_for(n, 128, 16);
    with_policy(blob, counts != nullptr, [&](auto policy) {
        using C = typename decltype(policy)::type;
        k_light_surfels<C><<<g, 128, blob_smem(blob, 128), st>>>(blob, s, n, evals, status, counts, terms);
    });
}

// kShared: many rows gather the cluster radiosities from shared memory, where
// a warp's 32 scattered 16-byte reads take some 10 cycles, a third of what
// they take in L1 (a cache line each).
template <bool kShared>
__global__ void __launch_bounds__(kJacBlock) k_jacobi_sell(const float4* direct, const float4* albedo,
                                                            float4* irr_out, float4* rad, uint32_t n, SellMatrix m,
                                                            const float4* __restrict__ crad, uint32_t nc,
                                                            SolveCtl* ctl, uint32_t it) {
    extern __shared__ __align__(16) uint8_t sell_smem[];
    pdl_wait();
    if (ctl->done) return;
    float4* cs = reinterpret_cast<float4*>(sell_smem);
    if constexpr (kShared) {
        for (uint32_t c = threadIdx.x; c < nc; c += blockDim.x) cs[c] = crad[c];
        __syncthreads();
    }
    float dmax = 0.0f;
    for (uint32_t sp = blockIdx.x * blockDim.x + threadIdx.x; sp < n; sp += gridDim.x * blockDim.x) {
        const uint32_t row = m.perm[sp];
        const V irr = kShared ? sell_row(m, cs, sp, m.len[sp]) : sell_row(m, crad, sp, m.len[sp]);
        dmax = fmaxf(dmax, row_update(direct, albedo, irr_out, rad, row, irr));
    }
    pdl_trigger();
    note_residual(dmax, ctl, it);
}

// One wave of CTAs, as many as are co-resident.
template <class K>
static unsigned wave_grid(K kernel, int block, size_t smem, unsigned long long items) {
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, smem);
    return grid_for(items, block, per_sm < 1 ? 1 : per_sm);
}

void launch_solve_bounce(cudaStream_t st, SurfelArrays s, uint32_t n, const float4* cp, const uint2* crange,
                         const uint32_t* members, uint32_t nc, const uint32_t* starts, const uint32_t* idx,
                         const float* w, float4* cluster_rad, SolveCtl* ctl, uint32_t it, int* launches,
                         int no_exit, const SellMatrix* sell) {
    launch_pdl(k_cluster_agg, nc < 4096u ? nc : 4096u, kAggBlock, 0, st, (const float4*)s.rad, (const float4*)s.p, cp,
               crange, members, nc, cluster_rad, ctl, it, no_exit);
    const float4 *direct = s.direct, *albedo = s.albedo, *crad = cluster_rad;
    const size_t cbytes = (size_t)nc * 16u;
    if (sell && sell->perm) {
        const bool many = n >= kManyRows && cbytes <= kSharedRadMax;
        const unsigned block = many ? (unsigned)kJacBlock : kFewRowsBlock;
        const unsigned grid = many ? wave_grid(k_jacobi_sell<true>, kJacBlock, cbytes, n) : grid_for(n, kFewRowsBlock);
        if ((many || cbytes <= kSharedRadSmall) && sell->links >= (uint64_t)grid * nc)
            launch_pdl(k_jacobi_sell<true>, grid, block, cbytes, st, direct, albedo, s.irr, s.rad, n, *sell, crad, nc, ctl,
                       it);
        else
            launch_pdl(k_jacobi_sell<false>, grid_for(n, kFewRowsBlock, 16), kFewRowsBlock, 0, st, direct, albedo, s.irr,
                       s.rad, n, *sell, crad, nc, ctl, it);
    } else if (n >= kWideRows && (((uintptr_t)idx | (uintptr_t)w) & 31u) == 0) {
        launch_pdl(k_jacobi_wide, grid_for(n, kJacBlock), kJacBlock, 0, st, direct, albedo, s.irr, s.rad, n, starts,
                   idx, w, crad, ctl, it);
    } else {
        const int vec = (((uintptr_t)idx | (uintptr_t)w) & 15u) == 0 ? 1 : 0;
        launch_pdl(k_jacobi, grid_for(n, kJacBlock), kJacBlock, 0, st, direct, albedo, s.irr, s.rad, n, starts, idx, w,
                   crad, ctl, it, vec);
    }
    *launches += 2;
}

void launch_solve_end(cudaStream_t st, SolveCtl* ctl, uint32_t it, int* launches) {
    launch_pdl(k_solve_end, 1u, 1u, 0, st, ctl, it);
    *launches += 1;
}

// ------------------------------------------------- sliced-ELL assembly ---
__global__ void k_sell_lens(const uint32_t* starts, uint32_t n, uint32_t* lens, uint32_t* rows) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        lens[i] = starts[i + 1] - starts[i];
        rows[i] = i;
    }
}

// Entries of slice k: 32 lanes x its longest row rounded up to 4 (rows are
// sorted by length, so that is the slice's first row).
__global__ void k_sell_sizes(const uint32_t* sorted_len, uint32_t n, uint32_t* sizes) {
    const uint32_t ns = (n + 31) / 32;
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k <= ns; k += gridDim.x * blockDim.x)
        sizes[k] = k < ns ? 32u * ((sorted_len[32 * k] + 3u) & ~3u) : 0u;
}

// A warp copies a slice, 32 links of each of its 32 rows at a time through
// shared memory: rows are read and the interleaved blocks written as whole
// lines. (A thread copying its own row touched a line per link on both sides:
// 0.226 ms for the 2.36M links of the Cornell box.)
static constexpr int kFillWarps = 4;
__global__ void __launch_bounds__(kFillWarps * 32) k_sell_fill(const uint32_t* starts, const uint32_t* idx,
                                                               const float* w, uint32_t n, const uint32_t* perm,
                                                               const uint32_t* sorted_len, const uint32_t* slice_off,
                                                               uint32_t* sidx, float* sw) {
    __shared__ uint32_t ti[kFillWarps][32][33];
    __shared__ float tw[kFillWarps][32][33];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t ns = (n + 31u) / 32u;
    for (uint32_t k = blockIdx.x * kFillWarps + warp; k < ns; k += gridDim.x * kFillWarps) {
        const uint32_t sp = k * 32u + lane;
        const uint32_t len = sp < n ? sorted_len[sp] : 0u, s0 = sp < n ? starts[perm[sp]] : 0u;
        const uint32_t base = slice_off[k], most = __shfl_sync(kFull, len, 0);
        for (uint32_t t = 0; t < most; t += 32u) {
#pragma unroll 8
            for (uint32_t r = 0; r < 32u; ++r) {
                const uint32_t sr = __shfl_sync(kFull, s0, r), lr = __shfl_sync(kFull, len, r);
                if (t + lane < lr) {
                    ti[warp][r][lane] = idx[(size_t)sr + t + lane];
                    tw[warp][r][lane] = w[(size_t)sr + t + lane];
                }
            }
            __syncwarp();
            // Four links of each row make a block of 128 entries.
            const uint32_t j0 = lane & 3u, blocks = min((most - t + 3u) / 4u, 8u);
            for (uint32_t q = 0; q < blocks; ++q)
#pragma unroll
                for (uint32_t r0 = 0; r0 < 32u; r0 += 8u) {
                    const uint32_t r = r0 + (lane >> 2), j = q * 4u + j0;
                    const size_t o = (size_t)base + ((t >> 2) + q) * 128u + r * 4u + j0;
                    if (t + j < __shfl_sync(kFull, len, r)) {
                        sidx[o] = ti[warp][r][j];
                        sw[o] = tw[warp][r][j];
                    }
                }
            __syncwarp();
        }
    }
}

int launch_sell_lens(cudaStream_t st, const uint32_t* starts, uint32_t n, uint32_t* lens, uint32_t* rows) {
    k_sell_lens<<<grid_for(n, 256), 256, 0, st>>>(starts, n, lens, rows);
    return 1;
}
int launch_sell_sizes(cudaStream_t st, const uint32_t* sorted_len, uint32_t n, uint32_t* sizes) {
    k_sell_sizes<<<grid_for((unsigned long long)(n + 31) / 32 + 1, 256), 256, 0, st>>>(sorted_len, n, sizes);
    return 1;
}
int launch_sell_fill(cudaStream_t st, const uint32_t* starts, const uint32_t* idx, const float* w, uint32_t n,
                     const uint32_t* perm, const uint32_t* sorted_len, const uint32_t* slice_off, uint32_t* sidx,
                     float* sw) {
    k_sell_fill<<<grid_for(n, kFillWarps * 32, 12), kFillWarps * 32, 0, st>>>(starts, idx, w, n, perm, sorted_len,
                                                                             slice_off, sidx, sw);
    return 1;
}

void configure_solve_kernels(int max_dyn_smem, bool no_grid) {
    for_each_policy(no_grid, [&](auto policy) {
        cudaFuncSetAttribute(k_light_surfels<typename decltype(policy)::type>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, max_dyn_smem);
    });
    cudaFuncSetAttribute(k_jacobi_sell<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSharedRadMax);
}

}  // namespace ifx
