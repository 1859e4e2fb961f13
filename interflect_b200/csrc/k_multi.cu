// Packed multi-scene frame: the solve of many independent scenes in one
// persistent cooperative launch and their shade in a second, both replayed
// from one graph (no counterpart in the reference, which renders one scene per
// process).
//
// Each scene was prepared through its own context: transfer, gather grid,
// per-surfel light factors (the emission-free terms of solve.rs:27-39) and
// one beauty frame whose hits, form factors and visibilities stay in that
// context's wavefront buffers. Per launch, for every scene at once:
//
//   relight   E_i = sum_l (rho_i * e_l) * a_il        (solve.rs:30-36)
//   bounce k  cluster means, Jacobi rows, per-scene stop rule
//                                                     (solve.rs:47-108)
//   refresh   the grid's copy of irr                  (surfel.rs:262-293)
//   compose   every pixel from its stored hits        (main.rs:289-358)
//
// Work items of all scenes are packed end to end (scene-major) and handed
// out grid-stride; the solve's phases are separated by a bounded grid barrier
// (its launch is cooperative, so every CTA is resident). The composition is a
// launch of its own: as a phase of the cooperative kernel it shared the
// bounces' 80 registers and one wave of CTAs over pixels of uneven cost
// (six scenes, 1.2M pixels: 2.51 -> 2.34 ms in all, and 1.94 ms
// with the rows read from the sliced-ELL copy). Every item performs
// exactly the operations of the single-scene kernels in the same order,
// so each scene is bit-identical to its own unbatched frame, whatever the
// packing, block size or grid.
#include "shade.cuh"

namespace ifx {

// Scene owning packed item `item`: the last scene whose base is <= item.
__device__ __forceinline__ int scene_of(const uint32_t* base, int S, uint32_t item) {
    int lo = 0, hi = S - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (base[mid] <= item) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// A cluster's members are summed by a warp, which loads 32 at a time, where
// there are so many a cluster in the mean, else by a thread: a warp takes as
// long for one member as for 32. Threads and warps, by scenes, members a cluster:
// 64 of 1.1 256 and 365 us, 16 of 4.4 383 and 436, 16 of 8.5 527 and 546, 6 of 25
// 835 and 688, 2 of 41 786 and 643.
static constexpr uint32_t kWarpMembers = 12;
// Scenes whose stop flags a CTA keeps in shared memory; the others' are formed
// anew for each item, from two words in L2. (All of them that way: 32 scenes of
// 300 surfels 375 us a frame with a warp per cluster, 355 with the flags.)
static constexpr int kStopFlags = 256;

__global__ void __launch_bounds__(256) k_multi_frame(MsParams M) {
    __shared__ uint8_t halted[kStopFlags];
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t stride = gridDim.x * blockDim.x;
    const MsScene* sc = M.scenes;

    // Relight, and reset the per-scene solve controls.
    for (uint32_t s = tid; s < (uint32_t)M.S; s += stride) M.ctl[s] = SolveCtl{};
    for (uint32_t item = tid; item < M.total_surf; item += stride) {
        const MsScene& S = sc[scene_of(M.surf_base, M.S, item)];
        const uint32_t i = item - S.surf_base;
        const V rho = mk4(S.albedo[i]);
        V out{0.0f, 0.0f, 0.0f};
        for (int l = 0; l < S.nl; ++l) {
            const float a = S.terms[(size_t)i * S.nl + l];
            if (a < 0.0f) continue;
            out = out + rho * mk4(S.lemit[l]) * a;
        }
        S.direct[i] = f4(out, 0.0f);
        S.rad[i] = f4(out, 0.0f);
        S.irr[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    if (!grid_barrier(M.bar, M.status, M.polls)) return;

    // The stop test of each bounce (solve.rs:93-101, with each scene's own
    // bounce cap) is part of the next one's first phase: every CTA forms it
    // from the residuals, CTA 0 also notes the scenes' statistics. `it` runs
    // one past the last bounce for that.
    for (uint32_t it = 0; it <= M.max_bounces; ++it) {
        auto stopped = [&](int s) {
            return solve_stopped<volatile SolveCtl>(M.ctl[s], it, 0) || it >= sc[s].max_bounces;
        };
        int live = 0;
        for (int s = (int)threadIdx.x; s < M.S; s += (int)blockDim.x) {
            const bool stop = stopped(s);
            live |= !stop;
            if (s < kStopFlags) halted[s] = stop;
            if (blockIdx.x == 0) solve_note(M.ctl[s], it, stop);
        }
        if (!__syncthreads_or(live)) break;
        auto over = [&](int s) { return s < kStopFlags ? halted[s] != 0 : stopped(s); };
        // solve.rs:61-73: cluster means, members summed in member order.
        const bool by_warps = M.total_surf / kWarpMembers >= M.total_clus;
        for (uint32_t item = tid; !by_warps && item < M.total_clus; item += stride) {
            const int s = scene_of(M.clus_base, M.S, item);
            if (over(s)) continue;
            const MsScene& S = sc[s];
            const uint32_t c = item - S.clus_base;
            const uint2 r = S.crange[c];
            V acc{0.0f, 0.0f, 0.0f};
            for (uint32_t k = r.x; k < r.y; ++k) {
                const uint32_t m = S.members[k];
                acc = acc + mk4(S.rad[m]) * S.sp[m].w;
            }
            S.crad[c] = f4(acc / fmaxf(S.cp[c].w, 1e-12f), 0.0f);
        }
        const uint32_t lane = threadIdx.x & 31u;
        for (uint32_t item = tid >> 5; by_warps && item < M.total_clus; item += stride >> 5) {
            const int s = scene_of(M.clus_base, M.S, item);
            if (over(s)) continue;
            const MsScene& S = sc[s];
            const uint32_t c = item - S.clus_base;
            const uint2 r = S.crange[c];
            V acc{0.0f, 0.0f, 0.0f};
            for (uint32_t k = r.x; k < r.y; k += 32u) {
                V v{0.0f, 0.0f, 0.0f};
                if (k + lane < r.y) {
                    const uint32_t m = S.members[k + lane];
                    v = mk4(S.rad[m]) * S.sp[m].w;
                }
                const uint32_t cnt = min(r.y - k, 32u);
                for (uint32_t j = 0; j < cnt; ++j)
                    acc = acc + V{__shfl_sync(kFull, v.x, j), __shfl_sync(kFull, v.y, j), __shfl_sync(kFull, v.z, j)};
            }
            if (lane == 0) S.crad[c] = f4(acc / fmaxf(S.cp[c].w, 1e-12f), 0.0f);
        }
        if (!grid_barrier(M.bar, M.status, M.polls)) return;
        // solve.rs:76-102: Jacobi rows; the residual is the per-scene max.
        for (uint32_t item = tid; item < M.total_surf; item += stride) {
            const int s = scene_of(M.surf_base, M.S, item);
            uint32_t bits = 0;  // this row's change as non-negative f32 bits (NaN ignored)
            if (!over(s)) {
                const MsScene& S = sc[s];
                // Rows in the order of their length, so that a warp's rows end
                // together and its loads are whole lines.
                const uint32_t sp = item - S.surf_base;
                const uint32_t i = S.sell.perm ? S.sell.perm[sp] : sp;
                const V irr = S.sell.perm ? sell_row(S.sell, S.crad, sp, S.sell.len[sp])
                                          : jacobi_row(S.crad, S.idx, S.w, S.starts[i], S.starts[i + 1], 1);
                V nr = mk4(S.direct[i]) + mk4(S.albedo[i]) * irr;
                V diff = vabs(nr - mk4(S.rad[i]));
                float d = fmaxf(diff.x, fmaxf(diff.y, diff.z));
                S.irr[i] = f4(irr, 0.0f);
                S.rad[i] = f4(nr, 0.0f);
                if (!isnan(d) && d > 0.0f) bits = __float_as_uint(d);
            }
            // One atomic per (warp, scene): the lanes of a scene reduce first.
            const unsigned grp = __match_any_sync(__activemask(), s);
            bits = __reduce_max_sync(grp, bits);
            if ((int)(threadIdx.x & 31) == __ffs(grp) - 1 && bits) atomicMax(&M.ctl[s].res[it & 1], bits);
        }
        if (!grid_barrier(M.bar, M.status, M.polls)) return;
    }

    // The grid's irradiance copy.
    for (uint32_t item = tid; item < M.total_surf; item += stride) {
        const MsScene& S = sc[scene_of(M.surf_base, M.S, item)];
        const uint32_t k = item - S.surf_base;
        S.girr[k] = S.irr[S.gitems[k]];
    }
}

// main.rs:289-358 for every pixel of every scene; nothing after a barrier
// that ran out.
__global__ void __launch_bounds__(128, 8) k_multi_compose(MsParams M) {
    if (*M.status) return;
    __shared__ float t8[256];
    for (int i = threadIdx.x; i < 256; i += blockDim.x) t8[i] = M.srgb_t[i];
    __syncthreads();
    NoCount cnt;
    for (uint32_t item = blockIdx.x * blockDim.x + threadIdx.x; item < M.total_pix; item += gridDim.x * blockDim.x) {
        const MsScene& S = M.scenes[scene_of(M.pix_base, M.S, item)];
        const SceneView sv = make_view(S.P.blob.ptr);
        const GatherView g = gview(S.P.grid);
        compose_pixel(sv, S.P, t8, g, item - S.pix_base, cnt);
    }
}

int launch_multi_frame(cudaStream_t st, const MsParams& p, int grid, int block) {
    void* args[] = {const_cast<MsParams*>(&p)};
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaLaunchKernelExC(&cfg, (const void*)k_multi_frame, args) != cudaSuccess) return -1;
    if (p.total_pix) k_multi_compose<<<grid_for(p.total_pix, 128, 64), 128, 0, st>>>(p);
    return 2;
}

int multi_frame_max_blocks(int block) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_multi_frame, block, 0) != cudaSuccess) return 0;
    return per_sm * sm_count();
}

}  // namespace ifx
