// bpc_dwt_plan.h -- access widths of the DWT's kernels (host side, no CUDA).
#pragma once
#include <stdint.h>

namespace bpc {

constexpr int kDwtThreads = 128;

// 16-byte accesses: both rasters 16-byte aligned, row stride and half a level's
// width multiples of 4 ints
inline bool dwt_vec4(const void *a, const void *b, int stride, int half) {
    return ((((uintptr_t)a) | ((uintptr_t)b)) & 15) == 0 && stride % 4 == 0 && half % 4 == 0;
}

// The copy of the odd levels' details: levels 1, 3, ... up to the returned one
// with 16-byte accesses (0: none), the deeper ones with 4-byte accesses.  A
// deeper level's half width divides a shallower one's, so a level that misfits
// leaves only those below it narrow, a sixteenth of the coefficients or less
// after level 1 (8256x6144, half of level 5 129 * 2, forward / inverse: all
// levels narrow 257 / 243 us, level 5 alone 172 / 157).
inline int dwt_copy_vec_level(const void *a, const void *b, int X, int levels) {
    int deepest = 0;
    for (int l = 1; l <= levels && dwt_vec4(a, b, X, (X >> (l - 1)) / 2); l += 2) deepest = l;
    return deepest;
}

// Columns of level 1 per CTA of that copy.  With level 1 wide, a narrow level
// (3 or deeper) has at most a quarter of its columns, so the same CTAs cover it.
inline int dwt_copy_columns(int vec_level) { return kDwtThreads * (vec_level >= 1 ? 4 : 1); }

}  // namespace bpc
