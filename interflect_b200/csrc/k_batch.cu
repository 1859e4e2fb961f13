// Batched relighting: R right-hand sides (emission vectors E^(r)) solved
// on one transfer matrix, the Jacobi bounce of solve.rs:47-108 as a CSR
// SpMM. Vectors are stored surfel-major with the R right-hand sides
// innermost (x[i * R + r], one float4 each), so a warp's lanes are 32
// right-hand sides of the same row: every load of a link's cluster value is
// one coalesced 512-byte access, and the link index and weight are
// warp-uniform. Each (row, rhs) accumulates its links in CSR order and each
// (cluster, rhs) its members in member order, exactly as the single-RHS
// kernels do, so every right-hand side is bit-identical to its own solve.
// Per-RHS done flags freeze a right-hand side at the bounce where its own
// residual fell below 1e-4 (solve.rs:99).
#include "kcommon.cuh"

namespace ifx {

// solve.rs:61-73 for every rhs: warp per (cluster, 32 rhs).
__global__ void __launch_bounds__(256) k_agg_batched(const float4* rad, const float4* sp, const float4* cp,
                                                      const uint2* crange, const uint32_t* members, uint32_t nc,
                                                      uint32_t R, float4* crad, const uint32_t* done) {
    const int lane = threadIdx.x & 31;
    const uint32_t chunks = (R + 31) / 32;
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < nc * chunks; t += warps) {
        const uint32_t c = t / chunks, r = (t % chunks) * 32 + lane;
        if (r >= R || done[r]) continue;
        const uint2 rg = crange[c];
        V acc{0.0f, 0.0f, 0.0f};
        uint32_t k = rg.x;
        for (; k + 8 <= rg.y; k += 8) {  // eight members' loads in flight
            float4 v[8];
            float a[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const uint32_t m = __ldg(&members[k + q]);
                v[q] = rad[(size_t)m * R + r];
                a[q] = __ldg(&sp[m].w);
            }
#pragma unroll
            for (int q = 0; q < 8; ++q) acc = acc + mk4(v[q]) * a[q];
        }
        for (; k < rg.y; ++k) {
            const uint32_t m = __ldg(&members[k]);
            acc = acc + mk4(rad[(size_t)m * R + r]) * __ldg(&sp[m].w);
        }
        crad[(size_t)c * R + r] = f4(acc / fmaxf(cp[c].w, 1e-12f), 0.0f);
    }
}

// solve.rs:76-102 for every rhs: blockIdx.y picks 32 rhs, warps stride over
// rows; a lane keeps its rhs for the whole kernel and reduces its residual
// to one integer atomicMax at the end.
__global__ void __launch_bounds__(512) k_spmm(const float4* direct, const float4* albedo, float4* irr, float4* rad,
                                               uint32_t n, uint32_t R, const uint32_t* starts, const uint32_t* idx,
                                               const float* w, const float4* crad, const uint32_t* done,
                                               uint32_t* res_bits) {
    const int lane = threadIdx.x & 31;
    const uint32_t r = blockIdx.y * 32 + lane;
    const bool live = r < R && !done[r];
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    float dmax = 0.0f;
    if (live) {
        for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += warps) {
            V acc{0.0f, 0.0f, 0.0f};
            const uint32_t e = starts[i + 1];
            for (uint32_t k = starts[i]; k < e; ++k)
                acc = acc + mk4(crad[(size_t)__ldg(&idx[k]) * R + r]) * __ldg(&w[k]);
            const size_t o = (size_t)i * R + r;
            const V nr = mk4(direct[o]) + mk4(__ldg(&albedo[i])) * acc;
            const V diff = vabs(nr - mk4(rad[o]));
            const float d = fmaxf(diff.x, fmaxf(diff.y, diff.z));
            irr[o] = f4(acc, 0.0f);
            rad[o] = f4(nr, 0.0f);
            if (!isnan(d)) dmax = fmaxf(dmax, d);
        }
        if (dmax > 0.0f) atomicMax(&res_bits[r], __float_as_uint(dmax));
    }
}

// The same with the cluster radiosities of kRhs right-hand sides in shared
// memory (12 bytes each: three arrays per cluster), kRhs lanes to a row. From
// global memory every link costs a warp 512 bytes of L1 or L2 and two uniform
// loads in a row before them; here it is three conflict-free reads and, as
// the row's links pass through a buffer of the warp (index and weight, 32 at
// a time), half a 16-byte broadcast. Each (row, rhs) still adds its links in
// CSR order. 16 right-hand sides, 12 bounces, Cornell box of 8,000, 20,000 and
// 60,000 surfels: 0.73 -> 0.61, 1.22 -> 1.01, 2.69 -> 1.95 ms.
static constexpr size_t kSpmmSharedMax = 200u * 1024u;
static constexpr uint32_t kRhs = 16;
static size_t spmm_shared_bytes(uint32_t nc, int warps) {
    return (size_t)nc * 3u * kRhs * 4u + (size_t)warps * 32u * 8u;
}

__global__ void __launch_bounds__(1024) k_spmm_shared(const float4* direct, const float4* albedo, float4* irr,
                                                      float4* rad, uint32_t n, uint32_t R, const uint32_t* starts,
                                                      const uint32_t* idx, const float* w, const float4* crad,
                                                      uint32_t nc, const uint32_t* done, uint32_t* res_bits) {
    extern __shared__ __align__(16) uint8_t spmm_smem[];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const uint32_t q = lane % kRhs, part = lane / kRhs, r = blockIdx.y * kRhs + q;
    const bool live = r < R && !done[r];
    if (!__syncthreads_or(live)) return;
    uint2* link = reinterpret_cast<uint2*>(spmm_smem) + warp * 32u + part * kRhs;
    float* cs = reinterpret_cast<float*>(spmm_smem + (size_t)warps * 32u * 8u);
    for (uint32_t e = threadIdx.x; e < nc * kRhs; e += blockDim.x) {
        const uint32_t c = e / kRhs, rr = blockIdx.y * kRhs + e % kRhs;
        const float4 v = rr < R ? crad[(size_t)c * R + rr] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        float* o = cs + (size_t)c * 3u * kRhs + e % kRhs;
        o[0] = v.x;
        o[kRhs] = v.y;
        o[2u * kRhs] = v.z;
    }
    __syncthreads();
    constexpr uint32_t kRows = 32u / kRhs;  // rows a warp takes together
    const uint32_t stride = gridDim.x * warps * kRows;
    float dmax = 0.0f;
    for (uint32_t i0 = (blockIdx.x * warps + warp) * kRows; i0 < n; i0 += stride) {
        const uint32_t i = i0 + part;
        uint32_t k = i < n ? starts[i] : 0u;
        const uint32_t e = i < n ? starts[i + 1] : 0u;
        V acc{0.0f, 0.0f, 0.0f};
        while (__any_sync(kFull, k < e)) {
            const uint32_t cnt = k < e ? min(e - k, kRhs) : 0u;
            // The cluster's place in shared memory, and the weight's bits.
            if (q < cnt) link[q] = make_uint2(__ldg(&idx[k + q]) * 3u * kRhs, __float_as_uint(__ldg(&w[k + q])));
            __syncwarp();
            uint32_t j = 0;
            for (; j + 4u <= cnt; j += 4u) {
                const uint4 a = *reinterpret_cast<const uint4*>(link + j), b = *reinterpret_cast<const uint4*>(link + j + 2);
                const float *c0 = cs + a.x + q, *c1 = cs + a.z + q, *c2 = cs + b.x + q, *c3 = cs + b.z + q;
                const V v0{c0[0], c0[kRhs], c0[2 * kRhs]}, v1{c1[0], c1[kRhs], c1[2 * kRhs]},
                    v2{c2[0], c2[kRhs], c2[2 * kRhs]}, v3{c3[0], c3[kRhs], c3[2 * kRhs]};
                acc = acc + v0 * __uint_as_float(a.y);
                acc = acc + v1 * __uint_as_float(a.w);
                acc = acc + v2 * __uint_as_float(b.y);
                acc = acc + v3 * __uint_as_float(b.w);
            }
            for (; j < cnt; ++j) {
                const uint2 a = link[j];
                const float* c = cs + a.x + q;
                acc = acc + V{c[0], c[kRhs], c[2 * kRhs]} * __uint_as_float(a.y);
            }
            __syncwarp();
            k += cnt;
        }
        if (i < n && live) {
            const size_t o = (size_t)i * R + r;
            const V nr = mk4(direct[o]) + mk4(__ldg(&albedo[i])) * acc;
            const V diff = vabs(nr - mk4(rad[o]));
            const float d = fmaxf(diff.x, fmaxf(diff.y, diff.z));
            irr[o] = f4(acc, 0.0f);
            rad[o] = f4(nr, 0.0f);
            if (!isnan(d)) dmax = fmaxf(dmax, d);
        }
    }
    if (dmax > 0.0f) atomicMax(&res_bits[r], __float_as_uint(dmax));
}

// Whether k_spmm_shared is the faster one for a matrix of so many rows and
// links. A CTA first copies all clusters, and a warp passes through its link
// buffer once more for each 16 links of a row: that pays from 32 links a row
// on, or half a million in all. Up to 32 warps a SM (from 530 clusters on one
// CTA) wait for a row's own loads and stores, which hides less than k_spmm's 64
// where these come from HBM: there from 60 links a row on. 8 bounces with
// k_spmm and shared, in us, by rows, clusters, mean links and right-hand sides:
//   6,000 x 779   117 links  16    472, 363      2,000 x 1,000   15 links  16    164, 193
//  45,000 x 809   119 links   2  1,664, 1,074   12,000 x 400      4 links  16    240, 300
// 110,000 x 225    34 links  10  3,222, 2,864  200,000 x 1,000   20 links  16  2,140, 3,422
// 120,000 x 500     5 links   1    733, 670    200,000 x 400     80 links  16  5,177, 4,638
// (the left column's first three are scenes' transfers). Over 1,323 matrices the
// rule costs 1% against the better one of each; k_spmm_shared for all costs 5%,
// and up to twice the time. It is wrong for up to 2,000 rows of like length and
// many links (2,000 x 300, 150 links: 257, 289), where scenes' transfers, whose
// longest rows are several times the mean, gain (2,000 x 862, 179 links: 455, 371).
static bool spmm_shared_wins(uint32_t n, uint32_t R, uint64_t links) {
    const uint64_t rows = n;
    if (links >= 60u * rows) return true;
    return rows * R <= 1250000u && (links >= 32u * rows || links >= (1u << 19));  // 80 MB an array
}

static void launch_spmm_shared(cudaStream_t st, const float4* direct, const float4* albedo, float4* irr, float4* rad,
                               uint32_t n, uint32_t R, const uint32_t* starts, const uint32_t* idx, const float* w,
                               const float4* crad, uint32_t nc, const uint32_t* done, uint32_t* res_bits, int warps) {
    const size_t sm = spmm_shared_bytes(nc, warps);
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_spmm_shared, warps * 32, sm);
    const unsigned chunks = (R + kRhs - 1u) / kRhs;
    const unsigned wave = (unsigned)sm_count() * (unsigned)(per_sm < 1 ? 1 : per_sm);
    const unsigned rows = (unsigned)warps * (32u / kRhs), need = (n + rows - 1u) / rows;
    const unsigned gx = wave / chunks < 1u ? 1u : wave / chunks;
    k_spmm_shared<<<dim3(gx < need ? gx : need, chunks), warps * 32, sm, st>>>(
        direct, albedo, irr, rad, n, R, starts, idx, w, crad, nc, done, res_bits);
}

// solve.rs:93-101 per rhs.
__global__ void k_bounce_end_batched(uint32_t R, uint32_t it, uint32_t* done, uint32_t* iterations,
                                     uint32_t* res_bits, uint32_t* last_res) {
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < R; r += gridDim.x * blockDim.x) {
        if (done[r]) continue;
        const float res = __uint_as_float(res_bits[r]);
        iterations[r] = it + 1;
        last_res[r] = res_bits[r];
        res_bits[r] = 0;
        if (res < 1e-4f) done[r] = 1;
    }
}

// E (R x n x 3 f32, rhs-major on the host side) -> direct = rad = E, irr = 0
// in the interleaved layout.
__global__ void k_batch_init(const float* E, uint32_t n, uint32_t R, float4* direct, float4* rad, float4* irr) {
    const size_t total = (size_t)n * R;
    for (size_t o = blockIdx.x * (size_t)blockDim.x + threadIdx.x; o < total; o += (size_t)gridDim.x * blockDim.x) {
        const size_t i = o / R, r = o % R;
        const float* e = E + (r * n + i) * 3;
        const float4 v = make_float4(e[0], e[1], e[2], 0.0f);
        direct[o] = v;
        rad[o] = v;
        irr[o] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
}

// Interleaved float4 -> rhs-major packed xyz.
__global__ void k_batch_unpack(const float4* x, uint32_t n, uint32_t R, float* out) {
    const size_t total = (size_t)n * R;
    for (size_t o = blockIdx.x * (size_t)blockDim.x + threadIdx.x; o < total; o += (size_t)gridDim.x * blockDim.x) {
        const size_t i = o / R, r = o % R;
        const float4 v = x[o];
        float* d = out + (r * n + i) * 3;
        d[0] = v.x;
        d[1] = v.y;
        d[2] = v.z;
    }
}

int launch_batch_init(cudaStream_t st, const float* E, uint32_t n, uint32_t R, float4* direct, float4* rad,
                      float4* irr) {
    k_batch_init<<<grid_for((unsigned long long)n * R, 256), 256, 0, st>>>(E, n, R, direct, rad, irr);
    return 1;
}

int launch_batch_unpack(cudaStream_t st, const float4* x, uint32_t n, uint32_t R, float* out) {
    k_batch_unpack<<<grid_for((unsigned long long)n * R, 256), 256, 0, st>>>(x, n, R, out);
    return 1;
}

int launch_batched_bounce(cudaStream_t st, uint32_t n, uint32_t R, const float4* sp, const float4* albedo,
                          const float4* direct, float4* irr, float4* rad, const float4* cp, const uint2* crange,
                          const uint32_t* members, uint32_t nc, const uint32_t* starts, const uint32_t* idx,
                          const float* w, float4* crad, uint32_t* done, uint32_t* iterations, uint32_t* res_bits,
                          uint32_t* last_res, uint32_t it, int rows_per_block_warps, uint64_t links) {
    const uint32_t chunks = (R + 31) / 32;
    k_agg_batched<<<grid_for((unsigned long long)nc * chunks * 32ull, 256), 256, 0, st>>>(rad, sp, cp, crange,
                                                                                          members, nc, R, crad, done);
    // Shared memory holds 16 right-hand sides of up to 1,024 clusters (192 bytes
    // each, beside 256 a warp: 1,056 at the smallest launch shape). With more
    // right-hand sides the warps of k_spmm are many and full, and lanes
    // whose right-hand side has converged cost it nothing: 256 of them on the
    // Cornell box's 20,000 surfels 6.1 ms against 9.3 in chunks of 16 (64:
    // 2.14 and 2.24; 24: 1.36 and 1.41).
    const int warps = 4 * rows_per_block_warps < 32 ? 4 * rows_per_block_warps : 32;
    if (R <= kRhs && spmm_shared_bytes(nc, warps) <= kSpmmSharedMax && spmm_shared_wins(n, R, links)) {
        launch_spmm_shared(st, direct, albedo, irr, rad, n, R, starts, idx, w, crad, nc, done, res_bits, warps);
    } else {
        const int block = 32 * rows_per_block_warps;
        unsigned gx = grid_for((unsigned long long)n * 32ull, block, 4);
        if (gx * chunks > 65535u * 64u) gx = (65535u * 64u) / chunks;
        dim3 grid(gx, chunks);
        k_spmm<<<grid, block, 0, st>>>(direct, albedo, irr, rad, n, R, starts, idx, w, crad, done, res_bits);
    }
    k_bounce_end_batched<<<grid_for(R, 256), 256, 0, st>>>(R, it, done, iterations, res_bits, last_res);
    return 3;
}

void configure_batch_kernels() {
    cudaFuncSetAttribute(k_spmm_shared, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSpmmSharedMax);
}

}  // namespace ifx
