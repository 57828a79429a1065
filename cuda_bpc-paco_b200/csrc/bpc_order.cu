// bpc_order.cu -- work order for images of several warp waves, and for the
// isolated decode of images of one or two waves.
//
// A CTA of the coder keeps its slot on the SM until its slowest warp is done,
// and the last wave of a launch runs on a partly idle GPU.  The time a warp
// spends on its codeblocks varies several-fold across an image (with the
// bitplanes coded and with how much the coder writes), so for images of many
// waves the coder is launched over the codeblocks sorted by expected work,
// heaviest first: warps of one CTA then get codeblocks of similar cost and
// the last wave holds the lightest ones.  The order changes only which warp
// codes which codeblock, never a stream word or a coefficient.
//
// Expected work of a work unit (the NG codeblocks one warp codes):
//   decoder: the slot words in use (MSB word + codewords), found by a search
//            for the first -1 of the fill (codewords are 0..0xFFFF; on a
//            damaged slot the search still ends inside it, and only the order
//            is affected), plus kPlaneWords per bitplane decoded;
//   encoder: the bitplanes coded, MSB + 1 (33 for an all-zero codeblock), from
//            all or, in a large image, every eighth row of the coefficients.
// The units are then counting-sorted by cost, descending (shared-memory atomics;
// units of equal cost in any order).
//
// An isolated decode (launch_code) takes the first units of the order for its
// heavy launch and hands the rest out from a queue counter that follows the
// order and the keys in the scratch; the sorting CTA zeroes it.
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

#include "bpc_kernels.h"

namespace bpc {

namespace {

constexpr int kBuckets = 1024;  // = threads of the sorting CTA
// decoder cost per plane in codeword-equivalents: a lockstep pass over a plane
// costs about as much as decoding 128 codewords (fit of per-codeblock decoder
// cycles on a B200 to words + planes).  For picking the few heaviest
// codeblocks of an isolated decode the planes weigh double: the chains that
// end last are those of the most planes (3-pass decodes with 64 / 128 / 256 /
// 512: 4096x4096 386 / 372 / 361 / 362 us, a noisy 5760x5760 690 / 667 / 629 /
// 630; 2 passes, 5120x5120 403 / 382 / 366 / 377).
constexpr uint32_t kPlaneWords = 128, kPlaneWordsIso = 256;

// Eight lanes per unit.  The first -1 is found eight probes at a time (four
// dependent loads) instead of by bisection, whose twelve were 9 us before a
// 4096x4096 decode could start; 32 probes at a time touch three times the
// sectors (16384x16384: 47 us).
template <int CBS>
__global__ void k_cost_dec(const int32_t *in, int ncb, uint32_t plane_words, uint32_t *key) {
    using G = Geo<CBS>;
    const int units = (ncb + G::NG - 1) / G::NG;
    const int lane = (int)(threadIdx.x & 31u), grp = lane >> 3, l8 = lane & 7;
    const int wstride = (int)(gridDim.x * blockDim.x) >> 5;
    for (int u4 = (int)(blockIdx.x * blockDim.x + threadIdx.x) >> 5; 4 * u4 < units; u4 += wstride) {
        const int u = 4 * u4 + grp;
        uint32_t cost = 0;
#pragma unroll
        for (int k = 0; k < G::NG; k++) {
            const int cb = u * G::NG + k;
            const bool ok = cb < ncb;
            const int32_t *slot = in + (size_t)(ok ? cb : 0) * (size_t)G::CAP;
            const int m = __ldg(slot);  // MSB word: planes decoded
            // words [lo, lo + 8 step) hold the first -1, if there is one; a
            // probe that reads a codeword moves lo behind it
            int lo = 0;
#pragma unroll
            for (int step = G::CAP / 8; step > 0; step = step > 1 && step < 8 ? 1 : step / 8) {
                const int i = lo + (l8 + 1) * step - 1;
                const bool used = i < G::CAP && __ldg(slot + (i < G::CAP ? i : 0)) != -1;
                const unsigned b = (__ballot_sync(0xffffffffu, used) >> (8 * grp)) & 0xFFu;
                lo += step * (__ffs((int)~b) - 1);
            }
            const uint32_t planes = m == 32 ? 33u : (m >= 0 && m <= 27 ? (uint32_t)m + 1u : 0u);
            if (ok) cost += (uint32_t)(lo < 1 ? 1 : lo) + plane_words * planes;
        }
        if (l8 == 0 && u < units) key[u] = cost;
    }
}

// The bitplanes of a codeblock from every ROWS-th of its rows.  Every eighth is
// enough to order the codeblocks of a large image (16384x16384: reading it
// whole took 150 us; the encode 3.94 -> 3.86 ms).  Up to kWholeCoeffs the whole
// image is read: what the L2 keeps of it the coder need not fetch again
// (2-pass encodes, whole / every eighth row: 6144x6144 0.395 / 0.425 ms, 8192x8192
// 0.677 / 0.703, 12288x12288 1.557 / 1.552).
constexpr long long kWholeCoeffs = 72ll << 20;
template <int CBS, int ROWS>
__global__ void k_cost_enc(const int32_t *in, int X, int ncbx, int ncb, uint32_t *key) {
    using G = Geo<CBS>;
    const int units = (ncb + G::NG - 1) / G::NG;
    const int lane = (int)(threadIdx.x & 31u), grp = lane / G::NL, gl = lane % G::NL;
    const int wstride = (int)(gridDim.x * blockDim.x) >> 5;
    for (int u = (int)(blockIdx.x * blockDim.x + threadIdx.x) >> 5; u < units; u += wstride) {
        const int cb = u * G::NG + grp;
        uint32_t mx = 0;
        if (cb < ncb) {
            const int cbx = cb % ncbx, cby = cb / ncbx;
            const int32_t *src = in + (size_t)cby * CBS * (size_t)X + (size_t)cbx * CBS + 2 * gl;
#pragma unroll 8
            for (int i = ROWS / 2; i < CBS; i += ROWS) {
                const int2 v = __ldg(reinterpret_cast<const int2 *>(src + (size_t)i * (size_t)X));
                mx |= (v.x < 0 ? 0u - (uint32_t)v.x : (uint32_t)v.x) | (v.y < 0 ? 0u - (uint32_t)v.y : (uint32_t)v.y);
            }
        }
        for (int o = G::NL / 2; o; o >>= 1) mx |= __shfl_xor_sync(0xffffffffu, mx, o);
        uint32_t cost = cb < ncb ? (mx ? 32u - (uint32_t)__clz((int)mx) : 33u) : 0u;
        if (G::NG == 2) cost += __shfl_xor_sync(0xffffffffu, cost, 16);
        if (lane == 0) key[u] = cost;
    }
}

// bin of a cost, descending: bin 0 holds the largest costs
__device__ __forceinline__ int cost_bin(uint32_t cost, int shift) {
    const uint32_t b = cost >> shift;
    return kBuckets - 1 - (int)(b > (uint32_t)(kBuckets - 1) ? (uint32_t)(kBuckets - 1) : b);
}

// Counting sort.  Every CTA counts the bins of all units, and apart from that
// those of the units before its own share, and so knows where its share goes
// without talking to the others; the loads of several rounds are in flight
// together.  The work grows with the square of the units, and so meets the sort
// on one CTA only at the largest image there is (encoder / decoder, one CTA ->
// this: 65,536 units 66 / 144 -> 38 / 17 us, 262,144 244 / 557 -> 130 / 43,
// 1,048,576, all that 2^31 - 1 coefficients hold, 953 / 2206 -> 964 / 266).
//
// COARSE (encoder, a few dozen different costs): a warp's units of equal cost
// claim their places together and stay in raster order.  Scattered one by one
// the same costs make a 6144x6144 encode 5 % slower (neighbouring codeblocks
// then run far apart).  The decoder's costs are nearly all different: it takes
// places one by one.
constexpr int kOrderAhead = 8, kOrderShare = 4 * kBuckets;
template <bool COARSE>
__global__ void __launch_bounds__(kBuckets) k_order(const uint32_t *key, int units, int shift, int ng, int *order,
                                                    int *ctr) {
    __shared__ uint32_t all[kBuckets], next[kBuckets];
    __shared__ uint32_t wsum[kBuckets / 32];
    const int tid = (int)threadIdx.x, lane = tid & 31;
    if (tid == 0 && blockIdx.x == 0 && ctr) *ctr = 0;  // the isolated decode's queue counter
    all[tid] = next[tid] = 0;
    __syncthreads();
    const int s0 = (int)blockIdx.x * kOrderShare, s1 = s0 + kOrderShare < units ? s0 + kOrderShare : units;
    // whole warps step through the units together (full-mask warp calls); s0
    // is a multiple of the warp's 32, so a warp's units lie on one side of it
    for (int u0 = tid - lane; u0 < units; u0 += kBuckets * kOrderAhead) {
        int bin[kOrderAhead];
#pragma unroll
        for (int k = 0; k < kOrderAhead; k++) {
            const int u = u0 + k * kBuckets + lane;
            bin[k] = u < units ? cost_bin(__ldg(key + u), shift) : -1;
        }
#pragma unroll
        for (int k = 0; k < kOrderAhead; k++) {
            uint32_t n = 1u;
            bool mine = bin[k] >= 0;
            if constexpr (COARSE) {
                const unsigned peers = __match_any_sync(0xffffffffu, bin[k]);
                n = (uint32_t)__popc(peers);
                mine = mine && lane == __ffs((int)peers) - 1;
            }
            if (mine) {
                atomicAdd(&all[bin[k]], n);
                if (u0 + k * kBuckets < s0) atomicAdd(&next[bin[k]], n);
            }
        }
    }
    __syncthreads();
    // exclusive scan of the bin counts
    const uint32_t v = all[tid];
    uint32_t x = v;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += t;
    }
    if (lane == 31) wsum[tid >> 5] = x;
    __syncthreads();
    if (tid < 32) {
        uint32_t y = wsum[tid];
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, y, o);
            if (lane >= o) y += t;
        }
        wsum[tid] = y;
    }
    __syncthreads();
    next[tid] += x - v + (tid >= 32 ? wsum[(tid >> 5) - 1] : 0u);
    __syncthreads();
    for (int r0 = s0; r0 < s1; r0 += kBuckets) {  // the whole CTA, round by round
        const int u = r0 + tid;
        const int bin = u < s1 ? cost_bin(__ldg(key + u), shift) : -1;
        if constexpr (COARSE) {
            const unsigned peers = __match_any_sync(0xffffffffu, bin);
            const int leader = __ffs((int)peers) - 1;
            uint32_t base = 0;
            if (bin >= 0 && lane == leader) base = atomicAdd(&next[bin], (uint32_t)__popc(peers));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (bin >= 0) order[base + (uint32_t)__popc(peers & ((1u << lane) - 1u))] = u * ng;
            __syncthreads();  // the rounds in order, too
        } else if (bin >= 0) {
            order[atomicAdd(&next[bin], 1u)] = u * ng;
        }
    }
}

}  // namespace

namespace {
// a device attribute, cached per device (callers may be on any host thread);
// 0 if it cannot be read
int cached_attr(cudaDeviceAttr a, std::atomic<int> *cache, int dev) {
    if (dev < 0 || dev >= 64) return 0;
    int n = cache[dev].load(std::memory_order_relaxed);
    if (!n) {
        if (cudaDeviceGetAttribute(&n, a, dev) != cudaSuccess || n <= 0) return 0;
        cache[dev].store(n, std::memory_order_relaxed);
    }
    return n;
}
}  // namespace

int sm_count(int dev) {
    static std::atomic<int> cache[64];
    return cached_attr(cudaDevAttrMultiProcessorCount, cache, dev);
}

int shared_optin(int dev) {
    static std::atomic<int> cache[64];
    return cached_attr(cudaDevAttrMaxSharedMemoryPerBlockOptin, cache, dev);
}

int shared_per_sm(int dev) {
    static std::atomic<int> cache[64];
    return cached_attr(cudaDevAttrMaxSharedMemoryPerMultiprocessor, cache, dev);
}

// warps resident at once on device `dev` (-1: the current device)
int resident_warps(bool enc, int dev) {
    if (dev < 0 && cudaGetDevice(&dev) != cudaSuccess) return 1 << 30;
    const int n = sm_count(dev);
    if (n <= 0) return 1 << 30;
    return n * kWarps * (enc ? kMinCtasEnc : kMinCtasDec);
}

namespace {

template <int CBS>
cudaError_t plan_t(bool enc, Params &p, int *sched, cudaStream_t st, bool iso) {
    using G = Geo<CBS>;
    const int units = (p.ncb + G::NG - 1) / G::NG;
    uint32_t *key = reinterpret_cast<uint32_t *>(sched + units);
    const uint32_t plane_words = iso ? kPlaneWordsIso : kPlaneWords;
    if (enc) {  // one warp per unit, grid-stride
        const int grid = (units + 7) / 8 < 4096 ? (units + 7) / 8 : 4096;
        if ((long long)p.X * p.Y <= kWholeCoeffs)
            k_cost_enc<CBS, 1><<<grid, 256, 0, st>>>(p.in, p.X, p.ncbx, p.ncb, key);
        else
            k_cost_enc<CBS, 8><<<grid, 256, 0, st>>>(p.in, p.X, p.ncbx, p.ncb, key);
    } else {
        const int grid = (units + 31) / 32 < 4096 ? (units + 31) / 32 : 4096;
        k_cost_dec<CBS><<<grid, 256, 0, st>>>(p.in, p.ncb, plane_words, key);
    }
    // bins of 2^shift cost units: decoder costs reach NG * (CAP + 33 * plane
    // words), encoder costs 2 * 33
    int shift = 0;
    if (!enc) {
        const long long mx = (long long)G::NG * ((long long)G::CAP + 33LL * plane_words);
        while ((mx >> shift) > kBuckets - 1) shift++;
    }
    int *ctr = iso ? sched + 2 * units : nullptr;
    const int ctas = (units + kOrderShare - 1) / kOrderShare;
    if (enc)
        k_order<true><<<ctas, kBuckets, 0, st>>>(key, units, shift, G::NG, sched, ctr);
    else
        k_order<false><<<ctas, kBuckets, 0, st>>>(key, units, shift, G::NG, sched, ctr);
    p.order = sched;
    p.ctr = ctr;
    return cudaGetLastError();
}

}  // namespace

long long sched_ints(int ncb, int cbs) {
    const int ng = cbs == 64 ? 1 : 2;
    // order and cost keys, one int each per unit, then the queue counter
    return 2LL * ((ncb + ng - 1) / ng) + 4;
}

bool order_pays(bool enc, int ncb, int cbs, int dev) {
    const int ng = cbs == 64 ? 1 : 2;
    // an image within two waves gains nothing from a balanced last wave: every
    // unit starts at once or in the second wave anyway
    return (long long)((ncb + ng - 1) / ng) >= 2LL * resident_warps(enc, dev);
}

cudaError_t plan_order(bool enc, int cbs, Params &p, int *sched, cudaStream_t st, bool isolate) {
    p.order = nullptr;
    p.ctr = nullptr;
    if (!sched || p.offsets || p.cb_begin != 0 || p.cb_end != p.ncb) return cudaSuccess;
    if (order_pays(enc, p.ncb, cbs))
        return cbs == 64 ? plan_t<64>(enc, p, sched, st, false) : plan_t<32>(enc, p, sched, st, false);
    // isolated decode: 64x64 codeblocks, more than nine tenths of a wave (below
    // that one-warp CTAs in raster order are faster: 3840x3840, 0.87 of a wave,
    // isolated / one-warp 0.362 / 0.352 ms in 3 passes, 0.251 / 0.246 in 2;
    // 4096x4096, 0.99, 0.345 / 0.376 and 0.251 / 0.248), more than the heavy
    // launch's share, and a device with SMs to spare for it
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return cudaSuccess;
    const long long res = resident_warps(false, dev);
    if (isolate && !enc && cbs == 64 && 10LL * p.ncb > 9 * res && p.ncb > 4 * kIsoCtas * kWarps &&
        sm_count(dev) > 4 * kIsoCtas && shared_optin(dev) > 0)
        return plan_t<64>(enc, p, sched, st, true);
    return cudaSuccess;
}

}  // namespace bpc
