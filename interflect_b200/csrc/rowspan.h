// Walking a row's links [s, e) eight at a time in 32-bit indices, where e may
// be as large as 2^32 - 1: sums such as k + 8 wrap there, so that the tests
// below compare differences. (A wrapped k + 8 <= e passes, reads past the
// arrays, and starts the row over at link 0 for ever.)
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define IFX_SPAN_FN __host__ __device__ __forceinline__
#else
#define IFX_SPAN_FN inline
#endif

namespace ifx {

static constexpr uint32_t kSpan = 8;

// Whether links [k, k + 8) all lie below e.
IFX_SPAN_FN bool span_full(uint32_t k, uint32_t e) { return k < e && e - k >= kSpan; }

// The place after k, which is below e; e if fewer than 8 links are left.
IFX_SPAN_FN uint32_t span_next(uint32_t k, uint32_t e) { return span_full(k, e) ? k + kSpan : e; }

}  // namespace ifx
