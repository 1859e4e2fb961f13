// The row walks of the solve's CSR kernels (interflect_b200/csrc/rowspan.h):
// for rows anywhere in 32-bit link indices, up to the very last, the walk ends,
// every full load lies inside the matrix, and each link of the row is taken
// once, in order. Both walks are checked: from the aligned place before the row
// (with the last links of the matrix one by one) and from a multiple of 4.
#include <cstdio>
#include <cstdint>

#include "../../interflect_b200/csrc/rowspan.h"

static int fail(const char* what, uint32_t s, uint32_t e, uint32_t total) {
    std::printf("%s: row [%u, %u) of %u links\n", what, s, e, total);
    return 1;
}

static int aligned_walk(uint32_t s, uint32_t e, uint32_t total) {
    uint64_t want = s;
    unsigned turns = 0;
    for (uint32_t k = s & ~(ifx::kSpan - 1u); k < e; k = ifx::span_next(k, e)) {
        if (++turns > 64) return fail("walk does not end", s, e, total);
        if (ifx::span_full(k, total)) {
            if ((uint64_t)k + ifx::kSpan > total) return fail("load past the matrix", s, e, total);
        } else {
            if ((uint64_t)k + ifx::kSpan <= total) return fail("links one by one that are not the last", s, e, total);
            for (uint32_t t = 0; t < ifx::kSpan; ++t)
                if ((uint64_t)k + t != (uint64_t)(uint32_t)(k + t)) return fail("index wraps", s, e, total);
        }
        if (k >= s && ifx::span_full(k, e)) {
            if (k != want) return fail("links out of order", s, e, total);
            want += ifx::kSpan;
            continue;
        }
        for (uint32_t t = 0; t < ifx::kSpan; ++t)
            if (k + t >= s && k + t < e) {
                if ((uint64_t)k + t != want) return fail("links out of order", s, e, total);
                ++want;
            }
    }
    return want == e ? 0 : fail("links left out", s, e, total);
}

static int plain_walk(uint32_t s, uint32_t e, uint32_t total) {
    uint64_t taken = 0;
    unsigned turns = 0;
    uint32_t k = s;
    for (; k < e && (k & 3u); ++k) ++taken;
    for (; ifx::span_full(k, e); k += ifx::kSpan) {
        if (++turns > 64) return fail("walk does not end", s, e, total);
        if ((uint64_t)k + ifx::kSpan > e) return fail("load past the row", s, e, total);
        taken += ifx::kSpan;
    }
    for (; k < e; ++k) ++taken;
    return taken == (uint64_t)e - s ? 0 : fail("links left out", s, e, total);
}

int main() {
    const uint32_t totals[] = {1u, 7u, 8u, 9u, 100u, 0x7fffffffu, 0x80000000u, 0xfffffff0u, 0xfffffff7u, 0xfffffff8u,
                               0xfffffff9u, 0xfffffffeu, 0xffffffffu};
    unsigned long long rows = 0;
    for (uint32_t total : totals)
        for (uint32_t back = 0; back <= 40 && back <= total; ++back)
            for (uint32_t len = 0; len <= 72; ++len) {
                const uint32_t e = total - back;
                if (len > e) continue;
                if (aligned_walk(e - len, e, total) || plain_walk(e - len, e, total)) return 1;
                ++rows;
            }
    std::printf("%llu rows walked to their ends\n", rows);
    return 0;
}
