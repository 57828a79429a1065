// bpc_dwt_plan.h -- access widths of the DWT's kernels (compiles without CUDA).
#pragma once
#include <stdint.h>

#if defined(__CUDACC__)
#define BPC_HD __host__ __device__
#else
#define BPC_HD
#endif

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
// levels narrow 249 / 235 us, level 5 alone 167 / 152).
inline int dwt_copy_vec_level(const void *a, const void *b, int X, int levels) {
    int deepest = 0;
    for (int l = 1; l <= levels && dwt_vec4(a, b, X, (X >> (l - 1)) / 2); l += 2) deepest = l;
    return deepest;
}

// Columns per CTA of that copy, four a thread in either access width: column j of
// thread t, side by side or a CTA's threads apart.  (One narrow column a thread
// kept too few loads in flight: 5998x4000, one level, forward / inverse 108 / 95
// -> 87 / 73 us; 8192x8192 off the 16-byte boundary, three levels, 365 / 317 -> 267
// / 222.)
constexpr int kDwtCopyColumns = 4 * kDwtThreads;
BPC_HD inline int dwt_copy_column(bool wide, int t, int j) {
    return wide ? 4 * t + j : (t / kDwtThreads) * kDwtCopyColumns + t % kDwtThreads + j * kDwtThreads;
}

}  // namespace bpc
