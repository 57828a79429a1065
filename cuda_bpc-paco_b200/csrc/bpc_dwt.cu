// bpc_dwt.cu -- reversible CDF 5/3 lifting DWT (JPEG 2000 integer filter) on
// the GPU, in the Mallat layout the coder's subband finder assumes: after each
// level the top-left (H >> l) x (W >> l) region holds [L | H] along x and
// [L ; H] along y.  Input and output are int32 rasters (the caller applies any
// DC level shift).  Symmetric extension: x[n] = x[n-2] for the predict step,
// d[-1] = d[0] for the update step; floor division by arithmetic shifts.
//
//   predict:  d[i] = x[2i+1] - floor((x[2i] + x[2i+2]) / 2)
//   update:   s[i] = x[2i]   + floor((d[i-1] + d[i] + 2) / 4)
//
// What bounds it: HBM traffic, and launches for small images.  One kernel does
// a level, rows and columns: a thread walks down a strip of 8 columns (4
// lifting pairs), lifts each row it reads in registers (the neighbours' samples
// by shuffle) and keeps the column lifting's state of those 8 values, so a
// level's region is read once and written once, with 16-byte accesses.  (A row
// kernel and a column kernel through the scratch moved it twice.)
//
// In place.  A level writes its four quadrants over rows other threads still
// read, so levels go out of place, in turn: level 1 data -> scratch, level 2
// scratch -> data (its details are then where they belong), level 3 data ->
// scratch, and so on; one copy kernel at the end brings the details of the odd
// levels back.  The inverse starts with that copy, the other way, and ends with
// level 1, scratch -> data.  Traffic per coefficient, 5 levels: 8 * 1.33 + 6.4
// = 17 B instead of 21 B, and 6 launches instead of 10.  B200, 5 levels, forward
// / inverse: 512x512 63 / 62 -> 35 / 35 us, 4096x4096 99 / 113 -> 72 / 66 us,
// 8192x6144 204 / 225 -> 166 / 155 us, 16384x16384 917 / 945 -> 765 / 715 us (6.0 /
// 6.4 TB/s over those 17 B).
#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdio>

#include "../../include/bpc_paco.h"
#include "bpc_dwt_plan.h"

namespace {

constexpr int kThreads = bpc::kDwtThreads;
constexpr unsigned kFull = 0xffffffffu;

// Vertical pairs per thread.  A strip reads 3 rows above its own again (from L2:
// its neighbour reads them at the same time); longer strips re-read less but
// leave the GPU idle at small levels (512x512 / 8192x6144 / 16384x16384 forward,
// 5 levels: 1 pair 36 / 168 / 793 us, 2: 35 / 166 / 765, 4: 40 / 172 / 773, 16,
// before chained launches: 91 / 231 / 796).
constexpr int kPairs = 2;


// Lets the next kernel of the call become resident, and waits for the one
// before to complete (returns at once in a plain launch).
__device__ __forceinline__ void after_previous() {
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <int N>
__device__ __forceinline__ void load_run(const int32_t *p, int32_t *v) {
    if constexpr (N % 4 == 0) {
#pragma unroll
        for (int k = 0; k < N; k += 4) {
            const int4 t = *reinterpret_cast<const int4 *>(p + k);
            v[k] = t.x, v[k + 1] = t.y, v[k + 2] = t.z, v[k + 3] = t.w;
        }
    } else {
#pragma unroll
        for (int k = 0; k < N; k++) v[k] = p[k];
    }
}
template <int N>
__device__ __forceinline__ void store_run(int32_t *p, const int32_t *v) {
    if constexpr (N % 4 == 0) {
#pragma unroll
        for (int k = 0; k < N; k += 4)
            *reinterpret_cast<int4 *>(p + k) = make_int4(v[k], v[k + 1], v[k + 2], v[k + 3]);
    } else {
#pragma unroll
        for (int k = 0; k < N; k++) p[k] = v[k];
    }
}

// P lifting pairs of a row per thread: 4 (16-byte accesses) or 1.  The strip
// starts at column c = 2 P (thread); lanes past the row's end (on = false) take
// part in the shuffles only.  v: the P low values, then the P high ones.
template <int P>
__device__ __forceinline__ void lift_row(const int32_t *row, int c, int w, bool on, int lane, int32_t v[2 * P]) {
    int32_t x[2 * P] = {}, xn = 0, xa = 0, xb = 0;
    if (on) {
        load_run<2 * P>(row + c, x);
        if (lane == 31 && c + 2 * P < w) xn = row[c + 2 * P];
        if (lane == 0 && c > 0) xa = row[c - 2], xb = row[c - 1];
    }
    const int32_t nb = __shfl_down_sync(kFull, x[0], 1);
    if (lane != 31) xn = nb;
    if (c + 2 * P >= w) xn = x[2 * P - 2];  // x[w] = x[w - 2]
    int32_t d[P];
#pragma unroll
    for (int k = 0; k < P; k++) d[k] = x[2 * k + 1] - ((x[2 * k] + (k + 1 < P ? x[2 * k + 2 < 2 * P ? 2 * k + 2 : 0] : xn)) >> 1);
    int32_t dp = __shfl_up_sync(kFull, d[P - 1], 1);
    if (lane == 0) dp = xb - ((xa + x[0]) >> 1);
    if (c == 0) dp = d[0];
#pragma unroll
    for (int k = 0; k < P; k++) {
        v[k] = x[2 * k] + ((dp + d[k] + 2) >> 2);
        v[P + k] = d[k];
        dp = d[k];
    }
}

// One level, rows then columns: the top-left w x h of `in` to the four
// quadrants of `out`, vertical pairs [blockIdx.y * kPairs, ...) per thread.
template <int P>
__global__ void __launch_bounds__(kThreads) k_fwd(const int32_t *in, int32_t *out, long long stride, int w, int h) {
    after_previous();
    const int c = (int)(blockIdx.x * kThreads + threadIdx.x) * 2 * P, lane = (int)(threadIdx.x & 31u);
    const bool on = c < w;
    const int hw = w >> 1, hh = h >> 1;
    const int i0 = (int)blockIdx.y * kPairs, i1 = i0 + kPairs < hh ? i0 + kPairs : hh;
    int32_t e[2 * P], dp[2 * P];  // row 2i, and the high values of pair i - 1
    if (i0 > 0) {
        int32_t a[2 * P], b[2 * P];
        lift_row<P>(in + (long long)(2 * i0 - 2) * stride, c, w, on, lane, a);
        lift_row<P>(in + (long long)(2 * i0 - 1) * stride, c, w, on, lane, b);
        lift_row<P>(in + (long long)(2 * i0) * stride, c, w, on, lane, e);
#pragma unroll
        for (int k = 0; k < 2 * P; k++) dp[k] = b[k] - ((a[k] + e[k]) >> 1);
    } else {
        lift_row<P>(in, c, w, on, lane, e);
    }
    int32_t *lo = out + (long long)i0 * stride + (c >> 1), *hi = lo + (long long)hh * stride;
#pragma unroll
    for (int i = i0; i < i1; i++) {
        int32_t o[2 * P], n[2 * P];
        lift_row<P>(in + (long long)(2 * i + 1) * stride, c, w, on, lane, o);
        if (2 * i + 2 < h) {
            lift_row<P>(in + (long long)(2 * i + 2) * stride, c, w, on, lane, n);
        } else {  // x[h] = x[h - 2]
#pragma unroll
            for (int k = 0; k < 2 * P; k++) n[k] = e[k];
        }
        int32_t s[2 * P], d[2 * P];
#pragma unroll
        for (int k = 0; k < 2 * P; k++) {
            d[k] = o[k] - ((e[k] + n[k]) >> 1);
            s[k] = e[k] + (((i == 0 ? d[k] : dp[k]) + d[k] + 2) >> 2);
            dp[k] = d[k];
            e[k] = n[k];
        }
        if (on) {
            store_run<P>(lo, s);
            store_run<P>(lo + hw, s + P);
            store_run<P>(hi, d);
            store_run<P>(hi + hw, d + P);
        }
        lo += stride;
        hi += stride;
    }
}

// One level back, columns then rows: the four quadrants of `in` to the top-left
// w x h of `out`.  The rows need values of the strips to the left and right
// that only come out of their column lifting, so the first and last lane of a
// warp work for their neighbours and store nothing (30 strips per warp).
template <int P>
__global__ void __launch_bounds__(kThreads) k_inv(const int32_t *in, int32_t *out, long long stride, int w, int h) {
    after_previous();
    const int lane = (int)(threadIdx.x & 31u);
    const int t = (int)(blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5)) * 30 + lane - 1;
    const int c = t * 2 * P;
    const bool on = c >= 0 && c < w, mine = on && lane > 0 && lane < 31;
    const int hw = w >> 1, hh = h >> 1;
    const int i0 = (int)blockIdx.y * kPairs, i1 = i0 + kPairs < hh ? i0 + kPairs : hh;
    const int32_t *lo = in + (c >> 1), *hi = lo + (long long)hh * stride;
    auto low = [&](int i, int32_t v[2 * P]) {
        if (!on) return;
        load_run<P>(lo + (long long)i * stride, v);
        load_run<P>(lo + (long long)i * stride + hw, v + P);
    };
    auto high = [&](int i, int32_t v[2 * P]) {
        if (!on) return;
        load_run<P>(hi + (long long)i * stride, v);
        load_run<P>(hi + (long long)i * stride + hw, v + P);
    };
    auto put_row = [&](int r, const int32_t v[2 * P]) {  // v: P low values, P high ones
        int32_t x[2 * P];
        int32_t dm = __shfl_up_sync(kFull, v[2 * P - 1], 1);
        if (c == 0) dm = v[P];
#pragma unroll
        for (int k = 0; k < P; k++) {
            x[2 * k] = v[k] - ((dm + v[P + k] + 2) >> 2);
            dm = v[P + k];
        }
        int32_t en = __shfl_down_sync(kFull, x[0], 1);
        if (c + 2 * P >= w) en = x[2 * P - 2];  // x[w] = x[w - 2]
#pragma unroll
        for (int k = 0; k < P; k++)
            x[2 * k + 1] = v[P + k] + ((x[2 * k] + (k + 1 < P ? x[2 * k + 2 < 2 * P ? 2 * k + 2 : 0] : en)) >> 1);
        if (mine) store_run<2 * P>(out + (long long)r * stride + c, x);
    };
    int32_t e[2 * P] = {}, d[2 * P] = {}, dm[2 * P] = {};
    low(i0, e);
    high(i0, d);
    if (i0 > 0) high(i0 - 1, dm);
#pragma unroll
    for (int k = 0; k < 2 * P; k++) e[k] -= ((i0 > 0 ? dm[k] : d[k]) + d[k] + 2) >> 2;
#pragma unroll
    for (int i = i0; i < i1; i++) {
        int32_t en[2 * P] = {}, dn[2 * P] = {}, o[2 * P];
        const bool more = i + 1 < hh;
        if (more) {
            low(i + 1, en);
            high(i + 1, dn);
        }
#pragma unroll
        for (int k = 0; k < 2 * P; k++) {
            en[k] = more ? en[k] - ((d[k] + dn[k] + 2) >> 2) : e[k];  // x[h] = x[h - 2]
            o[k] = d[k] + ((e[k] + en[k]) >> 1);
        }
        put_row(2 * i, e);
        put_row(2 * i + 1, o);
#pragma unroll
        for (int k = 0; k < 2 * P; k++) e[k] = en[k], d[k] = dn[k];
    }
}

// The details of levels 1, 3, ... (and, with whole, the low band of level
// `levels`) from one raster to the other.  blockIdx.y counts row groups of
// level 1, then of level 3, and so on.  Levels up to vec_level go with 16-byte
// accesses (dwt_copy_vec_level); WIDE / NARROW: some levels do / do not (both
// ways in every launch cost 3072x2048 1 us of 43).
constexpr int kCopyRows = 4;
template <bool WIDE>
__device__ __forceinline__ void copy_rows(const int32_t *in, int32_t *out, long long stride, int w, int h, int r0, int t,
                                          bool whole) {
    const int c0 = bpc::dwt_copy_column(WIDE, t, 0);
    int32_t v[kCopyRows][4];
    bool on[kCopyRows][4];
#pragma unroll
    for (int k = 0; k < kCopyRows; k++) {
        const int r = r0 + k;
        const int32_t *p = in + (long long)r * stride + c0;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int c = bpc::dwt_copy_column(WIDE, t, j);
            // the low quadrant belongs to the next level, unless this is the last
            on[k][j] = r < h && c < w && (whole || r >= (h >> 1) || c >= (w >> 1));
            if (!WIDE && on[k][j]) v[k][j] = p[j * kThreads];
        }
        if (WIDE && on[k][0]) load_run<4>(p, v[k]);
    }
#pragma unroll
    for (int k = 0; k < kCopyRows; k++) {
        int32_t *p = out + (long long)(r0 + k) * stride + c0;
        if (WIDE && on[k][0]) store_run<4>(p, v[k]);
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (!WIDE && on[k][j]) p[j * kThreads] = v[k][j];
    }
}
template <bool WIDE, bool NARROW>
__global__ void __launch_bounds__(kThreads) k_copy_odd(const int32_t *in, int32_t *out, long long stride, int X, int Y,
                                                       int levels, int vec_level) {
    after_previous();
    int y = (int)blockIdx.y, l = 1;
    for (; l <= levels; l += 2) {
        const int groups = ((Y >> (l - 1)) + kCopyRows - 1) / kCopyRows;
        if (y < groups) break;
        y -= groups;
    }
    if (l > levels) return;
    const int w = X >> (l - 1), h = Y >> (l - 1), t = (int)(blockIdx.x * kThreads + threadIdx.x);
    if (WIDE && (!NARROW || l <= vec_level))
        copy_rows<true>(in, out, stride, w, h, y * kCopyRows, t, l == levels);
    else
        copy_rows<false>(in, out, stride, w, h, y * kCopyRows, t, l == levels);
}

// Launch in stream order behind the level before it: its CTAs may become
// resident while that one drains and wait for it at their start
// (griddepcontrol.wait), which hides most of the launch latency (512x512 forward
// 46 -> 35 us, 8192x6144 175 -> 166 us).
template <class... P, class... A>
cudaError_t launch(bool chained, dim3 grid, cudaStream_t st, void (*kernel)(P...), A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(kThreads);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = chained ? 1 : 0;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
    if (e == cudaErrorNotSupported && cfg.numAttrs) {  // plain stream order then
        (void)cudaGetLastError();
        cfg.numAttrs = 0;
        e = cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
    }
    return e;
}

int check(cudaError_t e, const char *what) {
    if (e != cudaSuccess) {
        std::fprintf(stderr, "bpc dwt: %s: %s\n", what, cudaGetErrorString(e));
        return BPC_ERR_CUDA;
    }
    return BPC_OK;
}

bool valid(const int *d, const int *t, int X, int Y, int levels) {
    if (!d || !t || X <= 0 || Y <= 0 || levels < 0 || levels > 16) return false;
    // every level halves an even extent of at least 2
    return (X % (2 << (levels ? levels - 1 : 0))) == 0 && (Y % (2 << (levels ? levels - 1 : 0))) == 0 &&
           (X >> (levels ? levels - 1 : 0)) >= 2 && (Y >> (levels ? levels - 1 : 0)) >= 2 && X <= 32768 && Y <= 65535;
}

int level(bool fwd, bool chained, const int *in, int *out, int X, int Y, int l, cudaStream_t st) {
    const int w = X >> (l - 1), h = Y >> (l - 1);
    const unsigned gy = (unsigned)((h / 2 + kPairs - 1) / kPairs);
    const bool vec = bpc::dwt_vec4(in, out, X, w / 2);
    const int strips = vec ? w / 8 : w / 2, per = fwd ? kThreads : 30 * (kThreads / 32);
    const dim3 g((unsigned)((strips + per - 1) / per), gy);
    return check(launch(chained, g, st, fwd ? (vec ? k_fwd<4> : k_fwd<1>) : (vec ? k_inv<4> : k_inv<1>), in, out,
                        (long long)X, w, h),
                 "launch");
}

int copy_odd(bool chained, const int *in, int *out, int X, int Y, int levels, cudaStream_t st) {
    unsigned gy = 0;
    for (int l = 1; l <= levels; l += 2) gy += (unsigned)(((Y >> (l - 1)) + kCopyRows - 1) / kCopyRows);
    const int vec_level = bpc::dwt_copy_vec_level(in, out, X, levels), per = bpc::kDwtCopyColumns;
    const dim3 g((unsigned)((X + per - 1) / per), gy);
    const auto kernel = vec_level == 0 ? k_copy_odd<false, true>
                        : vec_level + 2 > levels ? k_copy_odd<true, false> : k_copy_odd<true, true>;
    return check(launch(chained, g, st, kernel, in, out, (long long)X, X, Y, levels, vec_level), "launch");
}

}  // namespace

extern "C" {

int bpc_dwt53_forward(int *d_data, int X, int Y, int levels, int *d_tmp, void *stream) {
    if (!valid(d_data, d_tmp, X, Y, levels)) return BPC_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    for (int l = 1; l <= levels; l++) {
        const int rc = level(true, l > 1, l % 2 ? d_data : d_tmp, l % 2 ? d_tmp : d_data, X, Y, l, st);
        if (rc) return rc;
    }
    return levels ? copy_odd(true, d_tmp, d_data, X, Y, levels, st) : BPC_OK;
}

int bpc_dwt53_inverse(int *d_data, int X, int Y, int levels, int *d_tmp, void *stream) {
    if (!valid(d_data, d_tmp, X, Y, levels)) return BPC_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    if (levels) {
        const int rc = copy_odd(false, d_data, d_tmp, X, Y, levels, st);
        if (rc) return rc;
    }
    for (int l = levels; l >= 1; l--) {
        const int rc = level(false, true, l % 2 ? d_tmp : d_data, l % 2 ? d_data : d_tmp, X, Y, l, st);
        if (rc) return rc;
    }
    return BPC_OK;
}

}  // extern "C"
