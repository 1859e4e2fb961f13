// Builds the object grid of a scene (objgrid.h), once per scene upload. No
// counterpart in the reference, which traverses its BVH for every query.
#include "kcommon.cuh"

#include <cuda_fp16.h>

namespace ifx {

// One CTA per block of 4 x 4 x 4 cells, a thread per cell. The CTA first
// keeps the objects that any of its cells can list (their distances at the
// block's centre, spread over the threads), then every cell tests those: the
// whole CTA evaluates the same object at a time, so the primitive code runs
// converged. A 512-object scene keeps some 30 objects per block.
static constexpr int kOgBlock = 64;

__global__ void __launch_bounds__(kOgBlock) k_og_build(BlobRef blob, ObjGrid g, OgLevel l, float lox, float loy,
                                                       float loz, float cell, uint32_t nbx, uint32_t nby,
                                                       uint32_t* mask, uint4* list, uint32_t* status) {
    IFX_SCENE_PROLOGUE(blob, status, sv);
    __shared__ uint32_t keep[kOgMaxObjects / 32];
    __shared__ float wmin[kOgBlock / 32];
    NoCount nc;
    const uint32_t nobj = (uint32_t)(sv.n_planes + sv.n_objects), words = (nobj + 31u) / 32u;
    const uint32_t b = blockIdx.x, t = threadIdx.x;
    const uint32_t bx = (b % nbx) * 4u, by = ((b / nbx) % nby) * 4u, bz = (b / (nbx * nby)) * 4u;
    const float half = og_half(cell, l.delta), bhalf = og_half(4.0f * cell, l.delta);
    {
        const V c{lox + (float)(bx + 2u) * cell, loy + (float)(by + 2u) * cell, loz + (float)(bz + 2u) * cell};
        float m = kMaxF;
        for (uint32_t i = t; i < nobj; i += kOgBlock) m = fminf(m, obj_dist(sv, sv.obj((int)i), c, nc));
        for (int o = 16; o >= 1; o >>= 1) m = fminf(m, __shfl_xor_sync(kFull, m, o));
        if ((t & 31u) == 0) wmin[t >> 5] = m;
        __syncthreads();
        m = fminf(wmin[0], wmin[1]);
        const float margin = og_margin(bhalf, l.delta) + og_margin(half, l.delta);
        for (uint32_t w = t >> 5; w < words; w += kOgBlock / 32) {
            const uint32_t i = w * 32u + (t & 31u);
            const bool in = i < nobj && og_listed(obj_dist(sv, sv.obj((int)(i < nobj ? i : 0u)), c, nc), m, margin);
            const uint32_t v = __ballot_sync(kFull, in);
            if ((t & 31u) == 0) keep[w] = v;
        }
        __syncthreads();
    }
    const uint32_t x = bx + (t & 3u), y = by + ((t >> 2) & 3u), z = bz + (t >> 4);
    const V p{lox + ((float)x + 0.5f) * cell, loy + ((float)y + 0.5f) * cell, loz + ((float)z + 0.5f) * cell};
    float m = kMaxF;
    for (uint32_t w = 0; w < words; ++w)
        for (uint32_t v = keep[w]; v; v &= v - 1u)
            m = fminf(m, obj_dist(sv, sv.obj((int)(w * 32u) + __ffs((int)v) - 1), p, nc));
    const float margin = og_margin(half, l.delta);
    uint32_t bits = 0, n = 0;
    float key[kOgListLen];
    uint32_t id[kOgListLen];
    for (uint32_t k = 0; k < kOgListLen; ++k) id[k] = 0, key[k] = 0.0f;
    for (uint32_t w = 0; w < words; ++w)
        for (uint32_t v = keep[w]; v; v &= v - 1u) {
            const uint32_t i = w * 32u + (uint32_t)__ffs((int)v) - 1u;
            const float d = obj_dist(sv, sv.obj((int)i), p, nc);
            if (!og_listed(d, m, margin)) continue;
            if (g.mode == kOgMask) {
                bits |= 1u << (i & 31u);
                continue;
            }
            uint32_t j = n < kOgListLen ? n : kOgListLen;
            for (; j > 0 && key[j - 1] > d; --j) {
                if (j == kOgListLen) continue;
                key[j] = key[j - 1];
                id[j] = id[j - 1];
            }
            if (j < kOgListLen) {
                key[j] = d;
                id[j] = i;
            }
            ++n;
        }
    if (x >= l.dim[0] || y >= l.dim[1] || z >= l.dim[2]) return;
    const uint32_t c = l.base + x + l.dim[0] * (y + l.dim[1] * z);
    if (g.mode == kOgMask) {
        mask[c] = bits;
        return;
    }
    const __half h = __float2half_rd(fminf(fmaxf(m, -60000.0f), 60000.0f));
    const float base = __half2float(h);
    uint32_t e[kOgListLen];
    for (uint32_t k = 0; k < kOgListLen; ++k) {
        e[k] = kOgNone;
        if (k >= n) continue;
        e[k] = n > kOgListLen && k == kOgListLen - 1 ? og_more(g.id_bits) : id[k];
        if (g.id_bits < 16) e[k] |= og_key(key[k], base, l.key_step) << g.id_bits;
    }
    list[c] = make_uint4((uint32_t)__half_as_ushort(h) | e[0] << 16, e[1] | e[2] << 16, e[3] | e[4] << 16,
                         e[5] | e[6] << 16);
}

void launch_og_build(cudaStream_t st, const BlobRef& blob, const ObjGrid& g, const OgLevel& l, const float lo[3],
                     float cell, uint32_t* mask, uint4* list, uint32_t* status) {
    const uint32_t nbx = (l.dim[0] + 3u) / 4u, nby = (l.dim[1] + 3u) / 4u, nbz = (l.dim[2] + 3u) / 4u;
    // The scene is read in place: nothing here waits, so no poll budget can
    // leave a grid half built, and the traversal stacks (at most 33 KiB) are
    // all its dynamic shared memory.
    BlobRef b = blob;
    b.staged = 0;
    k_og_build<<<nbx * nby * nbz, kOgBlock, blob_smem(b, kOgBlock), st>>>(b, g, l, lo[0], lo[1], lo[2], cell, nbx,
                                                                         nby, mask, list, status);
}

}  // namespace ifx
