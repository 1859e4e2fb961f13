// The object grid: for each cell of a uniform grid over the scene, the stored
// objects that can be nearest to a point of the cell. A distance query then
// evaluates one or two objects (over the CPU check's queries in the grid 1.2 are
// listed in the product and Cornell scenes, 1.5 in the 512-object stress scene)
// instead of traversing the BVH, and answers the reference's traversal exactly or says that it cannot.
//
// The rules, shared by the kernels and by the CPU check against the
// reference's traversal (tests/cpp/objgrid_check.cpp):
//
//  * Every admitted object's distance function is 1-Lipschitz and is nowhere
//    below the distance to its BVH leaf's box (leaf box distance 0 inside),
//    but for f32 rounding, which delta exceeds: a level's delta is 2^-16 of
//    the largest coordinate, length or radius in it plus the scene's diagonal,
//    about 32 times what eight roundings at that scale amount to. Where the
//    box's rounding alone matters a quarter of it is enough (the largest
//    shortfall found over 4e7 points of 16 scenes was 1/45 of delta).
//  * A cell lists every object whose distance at the cell's centre is at most
//    max(the nearest distance there, 0) + og_margin. An object that is not
//    listed is then, everywhere in the cell, farther than max(G, 0) + 3 delta,
//    G being the nearest distance at that point.
//  * A list carries a lower bound of each object's distance at the cell's
//    centre (og_key), and is sorted by it: a query stops at the first object
//    that cannot come within max(d1, 0) + delta of its point. A list too long
//    for its cell keeps the nearest objects and ends with the key of the next:
//    a query that gets there without stopping knows no answer.
//  * The query returns the smallest listed distance d1, its object o1, and d2,
//    the second smallest. If d2 > max(d1, 0) + delta/4, the reference's query
//    (bvh.rs:100-150: prune a node when its box distance >= the best so far,
//    objects by strict <) returns exactly (d1, o1): every other object is
//    farther than any box distance on o1's path in the tree, which is at most
//    max(d1, 0) plus rounding, so o1 cannot have been pruned, and no other
//    object is as near.
//  * A march that only stops at a surface needs no more than that the point is
//    inside: at d1 <= -delta the point is inside o1's box, so the reference
//    either evaluates o1 or pruned it against a best <= 0.
//  * At a near tie, the distance v1 to o1's leaf's box decides (the boxes on
//    o1's path are no farther): if d2 > v1 nothing can have pruned o1; if
//    v1 <= d1, only an object as near as o1 can. Planes are never pruned.
// Anything else (points outside the grid, ties within rounding of a box that
// both objects touch) asks the reference query.
//
// The same conditions let a cone-shadow march (trace.rs:84-124) skip queries:
// it advances 0.12 wherever the distance is at least that, and the distance
// changes by at most the step, so that a distance h guarantees the next
// (h - 0.12) / 0.12 steps.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define IFX_OG_FN __host__ __device__ __forceinline__
#else
#define IFX_OG_FN inline
#endif

namespace ifx {

// Two levels: the fine one over the scene's bounds, and one of coarse cells
// over eight times their extent, for the rays of a camera outside the bounds
// and those that leave them.
struct OgLevel {
    float inv;      // cells per unit length
    float bias[3];  // -lo * inv - 0.5: the cell index is the nearest integer to p * inv + bias
    uint32_t dim[3];
    uint32_t base;  // the level's first cell
    float delta;
    float side, key_step;  // the cells' side; what one unit of og_key stands for
};
struct ObjGrid {
    const uint32_t* mask;  // kOgMask: per cell, bit i = stored object i is listed
    // kOgList: per cell eight 16-bit words, the nearest distance at the centre
    // (half precision, rounded down), then up to kOgListLen objects, nearest
    // first: the stored-object index in the low id_bits, its og_key above.
    const uint32_t* list;
    OgLevel fine, coarse;
    int id_bits;           // 12, or 16 (and no keys) above kOgKeyObjects
    int mode;              // kOgOff, kOgMask, kOgList
};
static constexpr int kOgCoarseCells = 64;
static constexpr float kOgCoarseExtent = 8.0f;
enum : int { kOgOff = 0, kOgMask = 1, kOgList = 2 };
// Scenes of at most this many stored objects (planes and bounded) use masks.
static constexpr uint32_t kOgMaskObjects = 32;
static constexpr uint32_t kOgMaxObjects = 32768;
static constexpr uint32_t kOgKeyObjects = 4094;
static constexpr uint32_t kOgListLen = 7;
static constexpr uint32_t kOgNone = 0xffffu;  // end of a list
// The object index of a list's last word that stands for all that were left out: 2^id_bits - 2.
IFX_OG_FN uint32_t og_more(int id_bits) { return (1u << id_bits) - 2u; }

IFX_OG_FN uint32_t og_bits(float x) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(x);
#else
    uint32_t u;
    std::memcpy(&u, &x, 4);
    return u;
#endif
}

// One coordinate's cell: adding 2^23 rounds to the nearest integer, whose
// bits then follow from 2^23's. Negative, huge and NaN coordinates give an
// index no grid has.
IFX_OG_FN uint32_t og_axis(float p, float inv, float bias) {
    return og_bits(fmaf(p, inv, bias) + 8388608.0f) - 0x4B000000u;
}

// At least the distance of a point from its cell's centre: the parts of the
// cell index that og_axis rounds away, in cells' sides.
IFX_OG_FN float og_off_axis(float p, float inv, float bias) {
    const float f = fmaf(p, inv, bias);
    return f - ((f + 8388608.0f) - 8388608.0f);
}
IFX_OG_FN float og_from_centre(const OgLevel& l, float x, float y, float z) {
    const float a = og_off_axis(x, l.inv, l.bias[0]), b = og_off_axis(y, l.inv, l.bias[1]),
                c = og_off_axis(z, l.inv, l.bias[2]);
    return l.side * sqrtf(a * a + b * b + c * c) + 0.25f * l.delta;
}

// The key of an object at distance d from the centre of a cell whose nearest
// distance there is at least `base`: d is at least base + key * key_step.
IFX_OG_FN uint32_t og_key(float d, float base, float key_step) {
    const float k = (d - base) / key_step * (1.0f - 1e-6f);
    return k >= 15.0f ? 15u : (k > 0.0f ? (uint32_t)k : 0u);
}

// Whether an object of that key cannot come within max(d1, 0) + delta of a
// point `off` from the centre (an object's distance there is at least its
// distance at the centre less `off`).
IFX_OG_FN bool og_beyond(uint32_t key, float key_step, float base, float off, float d1, float delta) {
    return (float)key * key_step > fmaxf(d1, 0.0f) + 1.5f * delta + off - base;
}

IFX_OG_FN bool og_level_cell(const OgLevel& l, float x, float y, float z, uint32_t& cell) {
    const uint32_t i = og_axis(x, l.inv, l.bias[0]), j = og_axis(y, l.inv, l.bias[1]),
                   k = og_axis(z, l.inv, l.bias[2]);
    cell = l.base + i + l.dim[0] * (j + l.dim[1] * k);
    return i < l.dim[0] && j < l.dim[1] && k < l.dim[2];
}

// The cell of a point and which level it is of; false outside the grid.
IFX_OG_FN bool og_cell(const ObjGrid& g, float x, float y, float z, uint32_t& cell, bool& coarse) {
    coarse = false;
    if (og_level_cell(g.fine, x, y, z, cell)) return true;
    coarse = true;
    return og_level_cell(g.coarse, x, y, z, cell);
}

// Half-diagonal of a cube of side `side`, with room for the rounding of the
// cell index and of the centre.
IFX_OG_FN float og_half(float side, float delta) { return side * 0.8660255f + delta; }

// The listing margin over a cell of half-diagonal `half`: the nearest distance
// and an object's distance can each change by `half` between the centre and a
// point of the cell.
IFX_OG_FN float og_margin(float half, float delta) { return 2.0f * half + 4.0f * delta; }

// A level of `cells` cells along the longest side of [lo, hi] grown by `grow`
// about its centre; `scale` is the largest coordinate, length or radius of the
// scene's primitives. Returns the cell's side, and the level's corner in `from`.
inline double og_level(OgLevel& l, const float lo[3], const float hi[3], int cells, double grow, double scale,
                       double diag, uint32_t base, float from[3]) {
    double ext = 0.0;
    for (int a = 0; a < 3; ++a) ext = std::fmax(ext, (double)hi[a] - (double)lo[a]);
    const double side = ext * grow / cells;
    l.inv = (float)(1.0 / side);
    l.base = base;
    for (int a = 0; a < 3; ++a) {
        const double w = ((double)hi[a] - (double)lo[a]) * grow;
        const double f = ((double)lo[a] + (double)hi[a] - w) / 2.0;
        from[a] = (float)f;
        scale = std::fmax(scale, std::fmax(std::fabs(f), std::fabs(f + w)));
        l.bias[a] = (float)(-f / side - 0.5);
        const int n = (int)std::ceil(w / side);
        l.dim[a] = (uint32_t)(n < 1 ? 1 : (n > cells ? cells : n));
    }
    l.delta = (float)((scale + diag) / 65536.0);
    l.side = (float)side;
    l.key_step = og_margin(og_half(l.side, l.delta), l.delta) / 16.0f;
    return side;
}

IFX_OG_FN bool og_listed(float d, float nearest, float margin) { return !(d > fmaxf(nearest, 0.0f) + margin); }

// dist_only: the caller uses the distance to march and stops at any value
// <= 0 alike.
IFX_OG_FN bool og_exact(float d1, float d2, float delta, bool dist_only) {
    return d2 > fmaxf(d1, 0.0f) + 0.25f * delta || (dist_only && d1 <= -delta);
}

// og_exact at a near tie: v1 is the distance to o1's leaf's box.
IFX_OG_FN bool og_exact_box(float d1, float d2, float v1, bool dist_only) {
    return (d2 > v1 && d2 > d1) || (v1 <= d1 && (dist_only || d2 > d1));
}

// What a distance h at one point of a cone-shadow march says of the distance
// one 0.12 step on (rounding of the step, the position and h included), and
// what that says of the step after. The point is one of the grid, or one step
// from one: h is then no more than the distance from there to the objects, so
// that the points it speaks of lie within three times the coarse level's
// coordinates, and delta (the coarse level's) holds their rounding some ten
// times over. Outside the grid a coordinate can be as large as the caller
// likes, and nothing follows from h.
static constexpr float kOpenStep = 0.12f;
IFX_OG_FN float og_open_first(float h, float delta) { return h - 0.12002f - 4.0f * delta; }
IFX_OG_FN float og_open_next(float lower) { return lower - 0.12002f; }

}  // namespace ifx
