// bpc_core.cuh -- BPC-PaCo codeblock coder, one warp per 64x64 codeblock
// (two 16-lane groups per warp for 32x32 codeblocks).
//
// Bitstream contract (PabloEnfedaque/CUDA_BPC-PaCo, source/BPC_PaCo.cu):
//   * lane l of a codeblock owns the 2-column stripe at columns 2l, 2l+1 and
//     runs its own fixed-probability arithmetic coder (:261-339);
//   * planes b = MSB..0, passes SPP, MRP [, CP] (3-pass: an extra CP at MSB,
//     :968-1090), rows 0..H-1, left column then right column (:633-962);
//   * within one step all lanes make their significance/refinement call, then
//     the lanes that became significant make their sign call; an exhausted lane
//     reserves the next codeword slot in ascending lane order (__ballot/__popc,
//     :268-279).  That reservation order IS the bitstream.
//
// Representation (new): instead of one 32-bit word per coefficient with flag
// bits (:1120), a lane keeps bits of its stripe and of the two neighbour
// columns.  The encoder (bpc_enc.cuh) keeps words of 16 rows in scan order, both
// columns interleaved, and derives whole passes from them bit-parallel; the
// decoder (bpc_dec.cuh) walks the rows with a byte of neighbourhood bits per
// row.  Magnitudes are held as bitplanes in a per-thread array built with an
// in-register 32x32 bit transpose; the decoder collects decoded planes the same
// way and transposes them back at the end.  Shared memory holds the LUT bytes,
// the sign-context table and, per warp, the decoder's codeword window and row
// state or the encoder's event-ranking words and symbol descriptors.
//
// The code is written against a small warp interface W (lane id, ballot, any,
// shuffles, syncwarp) so the same source runs as a CUDA kernel (bpc_kernels.cu)
// and, compiled for the host with one user-level context per lane, in the CPU
// tests (tests/emu/emu_warp.cpp).
#pragma once
#include <stdint.h>

#if defined(__CUDACC__)
#define BPC_FI __device__ __forceinline__
#define BPC_NOINLINE __device__ __noinline__
#else
#define BPC_FI inline
#define BPC_NOINLINE inline
#endif

namespace bpc {

enum : int { ST_OVERFLOW = 1, ST_BAD_STREAM = 2, ST_INPUT_RANGE = 4, ST_LUT_RANGE = 8 };
enum : int { PK_SPP = 0, PK_MRP = 1, PK_CP = 2 };

// Sign-context table of Compute_Sign_Context (:178-211), indexed by
// (class(h) * 3 + class(v)), class = 0 for 0, 1 for > 0, 2 for < 0; 3 bits each.
constexpr uint32_t kSignTab = (0u << 0) | (2u << 3) | (3u << 6) | (4u << 9) | (6u << 12) | (0u << 15) |
                              (5u << 18) | (1u << 21) | (7u << 24);

// The decoder's sign-context table.  The four neighbours a left-column
// coefficient's sign depends on sit at kSignBits of its 3-row window
// (bpc_dec.cuh; up 1, left 8, right 10, below 17, their signs 4 bits above);
// multiplied by kSignHash the 256 combinations differ in the top byte, the
// table's index (found by search; test_sign_hash_is_perfect checks it).  An
// entry is the byte-permute selector that picks the LUT probability (ctx >> 1)
// out of a word of four, zero-extended, with the predicted sign (ctx & 1) in
// bit 15 (which selects a zero byte either way).  Threads tid, tid + n, ...
// fill it.
// The eight neighbours of a significance context are at kCtxBits.
constexpr uint32_t kCtxBits = 0x00070507u, kSignBits = 0x00225522u, kSignHash = 0x01040400u;
constexpr int kSignTableBytes = 512;
BPC_FI void build_sign_table(uint8_t *table, int tid, int n) {
    uint16_t *t = reinterpret_cast<uint16_t *>(table);
    for (int k = tid; k < kSignTableBytes / 2; k += n) {
        const int sl = k & 1, nl = (k >> 1) & 1, sr = (k >> 2) & 1, nr = (k >> 3) & 1;
        const int su = (k >> 4) & 1, nu = (k >> 5) & 1, sb = (k >> 6) & 1, nb = (k >> 7) & 1;
        const int h = sl * (1 - 2 * nl) + sr * (1 - 2 * nr), v = su * (1 - 2 * nu) + sb * (1 - 2 * nb);
        const int hc = h == 0 ? 0 : (h > 0 ? 1 : 2), vc = v == 0 ? 0 : (v > 0 ? 1 : 2);
        const uint32_t ctx = (kSignTab >> (3 * (hc * 3 + vc))) & 7u;
        const uint32_t window = (uint32_t)su << 1 | (uint32_t)nu << 5 | (uint32_t)sl << 8 | (uint32_t)nl << 12 |
                                (uint32_t)sr << 10 | (uint32_t)nr << 14 | (uint32_t)sb << 17 | (uint32_t)nb << 21;
        t[(window * kSignHash) >> 24] = (uint16_t)(0x4440u | (ctx >> 1) | ((ctx & 1u) << 15));
    }
}

// Eight 0-symbols of probability P from interval size sz: the size after them,
// and before the last one (0: the codeword was used up before).
BPC_FI void zero_run(uint32_t &sz, uint32_t &prev, uint32_t P) {
    prev = sz;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        prev = sz;
        sz = (sz * P) >> 7;
    }
}
// 0-symbols until size sz is used up, at most 8
BPC_FI int zero_count(uint32_t sz, uint32_t P) {
    int n = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        n += sz != 0u ? 1 : 0;
        sz = (sz * P) >> 7;
    }
    return n;
}

struct Params {
    const int32_t *in;   // encode: raster coefficients; decode: slot stream
    int32_t *out;        // encode: slot stream; decode: raster coefficients
    const int32_t *lut;  // loader array (ints)
    int lut_n;           // its length
    int tab_n;           // shared byte table length (covers every index the coder forms)
    int X, Y, levels;
    int ncbx, ncb;       // codeblocks per row, total
    int a_sig, a_sign, cp_off;  // LUT section offsets as the reference kernel forms them
    int *status;         // OR of ST_* bits, may be null
    int *counts;         // per-codeblock codeword count, may be null
    // decoder input in the compact container: codeblock k's words (MSB and
    // codewords) are in[offsets[k] .. offsets[k+1]); null = slot layout
    const long long *offsets;
    long long in_words = 0;  // compact container: its length in words (offsets outside it are damage)
    int cb_begin, cb_end;  // codeblocks [cb_begin, cb_end) of the image are coded by this launch
    // work order of a whole-image launch: warp slot k codes the codeblocks
    // starting at order[k] (null = raster order)
    const int *order = nullptr;
    // isolated decode of a work-ordered image (launch_code): heavy = 1 codes
    // the units order[0, heavy_n), one per warp slot; heavy = 2 codes the rest,
    // one unit per warp slot first and then units taken from the queue counter
    // *ctr (zeroed by the planner).  heavy = 0: the plain grid-stride walk.
    int heavy = 0, heavy_n = 0;
    int *ctr = nullptr;
};

// LUT offsets the reference kernel uses (Initialize_LUT_pointers :228-250 with
// LUT_N_BITPLANES = 15, and the CP offset :988-989).  tab_n, the bytes of table
// a kernel keeps, depends on the mode alone (at most 19,920, at 16 levels and 3
// passes): entries of a longer LUT that the coder cannot index are range-checked
// and not kept, so the shared memory of a launch does not grow with the LUT.
struct LutOffsets {
    int a_sig, a_sign, cp_off, tab_n;
};
inline LutOffsets lut_offsets(int levels, int passes, int /*lut_n*/) {
    LutOffsets o;
    const int ref_n = 3 * 15 * 1 * levels + 15 * 1;
    const int sig_n = 3 * 15 * 9 * levels + 15 * 9;
    const int sign_n = 3 * 15 * 4 * levels + 15 * 4;
    o.a_sig = ref_n;
    o.a_sign = ref_n + sig_n;
    o.cp_off = sig_n + sign_n;
    // largest index formed: LL group (levels*45) at plane 32 (all-zero block)
    const int gmax = levels * 45 + 32;
    int mx = gmax;  // refinement
    int s1 = o.a_sig + gmax * 9 + 8, s2 = o.a_sign + gmax * 4 + 3;
    if (passes == 3) {
        s1 += o.cp_off;
        s2 += o.cp_off;
    }
    mx = mx > s1 ? mx : s1;
    mx = mx > s2 ? mx : s2;
    o.tab_n = (mx + 1 + 15) & ~15;
    return o;
}

template <int CBS>
struct Geo {
    static constexpr int NL = CBS / 2;                   // lanes per codeblock
    static constexpr int NG = 32 / NL;                   // codeblocks per warp
    static constexpr int CAP = CBS * CBS;                // slot size in ints
    static constexpr int RING = CBS == 64 ? 512 : 256;   // decoder: codeword window per codeblock
    static constexpr int CHUNK = RING / 2;               // words a refill moves the window on
    // decoder state of a warp in shared memory (bpc_dec.cuh): row bytes,
    // refinement sets, SPP-coded marks
    static constexpr int ROW_WORDS = CBS / 4 * 32, REF_WORDS = CBS / 16 * 32, VIS_WORDS = CBS / 4 * 8;
    static constexpr int RING_WORDS = RING * NG + ROW_WORDS + REF_WORDS + VIS_WORDS;  // per warp
};

BPC_FI int popc32(uint32_t x) {
#if defined(__CUDA_ARCH__)
    return __popc(x);
#else
    return __builtin_popcount(x);
#endif
}
BPC_FI void add_u64(unsigned long long *p, unsigned long long v) {
#if defined(__CUDA_ARCH__)
    atomicAdd(p, v);
#else
    *p += v;
#endif
}
BPC_FI int ctz32(uint32_t x) {
#if defined(__CUDA_ARCH__)
    return __ffs((int)x) - 1;
#else
    return __builtin_ctz(x);
#endif
}
BPC_FI uint32_t brev32(uint32_t x) {
#if defined(__CUDA_ARCH__)
    return __brev(x);
#else
    uint32_t r = 0;
    for (int k = 0; k < 32; k++) r |= ((x >> k) & 1u) << (31 - k);
    return r;
#endif
}
BPC_FI int clz32(uint32_t x) {
#if defined(__CUDA_ARCH__)
    return __clz(x);
#else
    return x ? __builtin_clz(x) : 32;
#endif
}

// In-register transpose of a 32x32 bit matrix, LSB first: afterwards bit r of
// a[c] is what bit c of a[r] was.  (Recursive block swap; 5 x 16 exchanges.)
BPC_FI void transpose32(uint32_t a[32]) {
    uint32_t m = 0x0000FFFFu;
#pragma unroll
    for (int j = 16; j; j >>= 1, m ^= m << j) {
#pragma unroll
        for (int k = 0; k < 32; k = (k + j + 1) & ~j) {
            const uint32_t t = ((a[k] >> j) ^ a[k + j]) & m;
            a[k + j] ^= t;
            a[k] ^= t << j;
        }
    }
}

BPC_FI uint32_t funnel_r(uint32_t lo, uint32_t hi, int n) {
#if defined(__CUDA_ARCH__)
    return __funnelshift_r(lo, hi, n);
#else
    return (uint32_t)((((uint64_t)hi << 32) | lo) >> (n & 31));
#endif
}

// byte selectors sel (four 4-bit digits, 0-3: bytes of v, 4-7: zero)
BPC_FI uint32_t perm8(uint32_t v, uint32_t sel) {
#if defined(__CUDA_ARCH__)
    return __byte_perm(v, 0u, sel);
#else
    uint32_t r = 0;
    for (int k = 0; k < 4; k++) {
        const uint32_t d = (sel >> (4 * k)) & 7u;
        r |= (d < 4u ? (v >> (8 * d)) & 0xFFu : 0u) << (8 * k);
    }
    return r;
#endif
}

// Size of the encoder's per-lane event array (8-byte aligned): two words per
// reservation of one pass.  There is at most one reservation per symbol call,
// and a lane makes at most two calls per coefficient of its stripe (256 for
// 64x64, 128 for 32x32).  kEvKeys: the constructor's byte array, which no coder
// uses any more.
constexpr int kEvKeys = 1, kEvVals = 512;

// Decoder codeword window: lane gl of a codeblock's lane group fills its share
// of the window with slot words [first, first + RING), 16-byte loads where it
// can; words past in_cap read as -1.  (The words of the window's second half
// move to its first half through memory again: they are in L2 or L1, and this
// runs once per 256 codewords.)  Kept out of line: inlined into every decoder
// step body it would crowd the instruction cache.
// All loads are issued before the first word is stored, so a refill waits for
// memory once and not four times (a codeblock decoded alone refills up to eight
// times: 186 -> 178 us, 2 passes).
template <int CBS>
BPC_NOINLINE void ring_fill(uint32_t *ring, const int32_t *slot_in, uint32_t in_cap, bool compact, uint32_t first,
                            int gl) {
    using G = Geo<CBS>;
    constexpr int per = G::RING / G::NL;  // 16, a multiple of 4
    uint32_t v[per];
#pragma unroll
    for (int q = 0; q < per; q += 4) {
        const uint32_t k = first + (uint32_t)(q * G::NL + 4 * gl);
        if (k + 3 < in_cap && !compact) {
#if defined(__CUDA_ARCH__)
            const int4 t = __ldg(reinterpret_cast<const int4 *>(slot_in + k));
            v[q] = (uint32_t)t.x;
            v[q + 1] = (uint32_t)t.y;
            v[q + 2] = (uint32_t)t.z;
            v[q + 3] = (uint32_t)t.w;
#else
            for (int i = 0; i < 4; i++) v[q + i] = (uint32_t)slot_in[k + i];
#endif
        } else {  // slot end, or the compact container (no 16-byte alignment)
#pragma unroll
            for (int i = 0; i < 4; i++) v[q + i] = k + i < in_cap ? (uint32_t)slot_in[k + i] : 0xFFFFFFFFu;
        }
    }
#pragma unroll
    for (int q = 0; q < per; q++) ring[(q & ~3) * G::NL + 4 * gl + (q & 3)] = v[q];
}

// LAT > 0 selects the decoder's latency form, for launches whose time is the
// serial chain of their heaviest codeblocks rather than the SMs' issue rate: a
// step reads its sign context before its significance decision (more
// instructions, the same bitstream).  The encoder has one form.
// Coder<..., ENC = true> is in bpc_enc.cuh, ENC = false in bpc_dec.cuh.
template <int PASSES, int CBS, bool ENC, class W, int LAT = 0>
struct Coder;

// Find_Subband :84-111 for a lane's column x and the codeblock's top row y0:
// first LUT plane of its level and subband
BPC_FI int lut_group(const Params &p, int x, int y0) {
    int lvl = p.levels, sb = 0;
    for (int a = 1; a <= p.levels; a++) {
        const bool hx = x >= (p.X >> a), hy = y0 >= (p.Y >> a);
        if (hx || hy) {
            lvl = a - 1;
            sb = hx ? (hy ? 2 : 0) : 1;
            break;
        }
    }
    return lvl * 45 + sb * 15;
}

}  // namespace bpc

#include "bpc_dec.cuh"
#include "bpc_enc.cuh"
