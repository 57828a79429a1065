// bpc_enc.cuh -- the BPC-PaCo codeblock encoder (included by bpc_core.cuh).
//
// What bounds it: integer issue in the per-lane symbol loop, and for an image
// of a wave or two the serial chain of the heaviest codeblocks.  The encoder
// knows every data bit, so per pass it finds bit-parallel which coefficients
// are coded (K), which code a 1 and become significant (NS) and all their
// contexts, time-accurate (neighbours earlier in scan order: start of pass |
// NS; later: start of pass).  Each lane then runs its arithmetic coder over its
// own coded symbols only.  A reservation (:268-279) is recorded as an event keyed
// by (row, column, phase); at the end of the pass the warp ranks the events by
// (key, lane) -- the reference's lockstep order -- and the codewords go to
// their slots.
//
// Layout.  A lane's stripe is NQ words of 16 rows: bit 2r + c is row r, column
// c, which is the scan order, so a word of K is walked with one find-first per
// symbol.  The neighbour columns share one word in the same places: the outer
// neighbour of a left coefficient is lane-1's right column (even bits), of a
// right one lane+1's left column (odd bits); the inner neighbour is the
// adjacent bit, the rows above and below are shifts by two.
//
// A word's eight slices (four of the context, the symbol, two of the sign
// context, the sign symbol) are transposed into one descriptor byte per
// position in shared memory, 56 instructions for 32 positions, instead of being
// picked apart bit by bit for every symbol (about 20 each).  The loop reads the
// next position's descriptor and probability while it codes this one (serial
// chain of one LL codeblock alone: 203 -> 177 us), and an event is one 8-byte
// store (171 -> 150 us).  One call per loop iteration, the sign call as the next
// one, measured no faster over large images and slower on that chain (159 us).
//
// B200, against column masks with zipped slices and all-zero codeblocks coded
// like any other: 16384x16384 3-pass encode 6.68 -> 3.93 ms, 4096x4096 0.42-0.75
// -> 0.33 ms (the slow end: 15 all-zero codeblocks), 2048x2048 2-pass 0.152 ->
// 0.127 ms.
#pragma once

namespace bpc {

template <int PASSES, int CBS, class W, int LAT>
struct Coder<PASSES, CBS, true, W, LAT> {
    using G = Geo<CBS>;
    static constexpr int NQ = CBS / 16;  // words per stripe
    static constexpr uint32_t EV = 0x55555555u, OD = 0xAAAAAAAAu;
    W &w;
    const Params &p;
    const uint8_t *tab;  // LUT bytes
    int32_t *slot_out;
    uint32_t *evmask;  // per warp, 256 keys: lanes with a reservation event
    uint32_t *pfx;     // per warp, 256 words: events before the key (ranking); descriptors of the symbol loop
    // this lane's events of the pass, two words each: the coder's L then (the
    // value of the codeword before, plus 1), and the key
    uint32_t *ev;
    // magnitude bitplanes, [plane][word] (a per-thread array owned by the caller)
    uint32_t (*planes)[4];
    int lane, gl, g, msb, status;
    int top;        // highest bitplane coded from the stored planes (-1: none)
    uint32_t qtop;  // byte q = 1 + the highest plane stored for word q (0: none)
    uint32_t gmask, ltmask;
    uint32_t mL, mR;  // EV / OD, or 0 at the codeblock's left / right edge
    // arithmetic coder: Lower = L - 1, Size = E - L
    uint32_t L, E;
    uint32_t cnt;   // codewords reserved in this codeblock (group-uniform)
    int open_slot;  // slot of the lane's last reservation (-1: none yet)
    int nev;        // events of the pass
    // LUT statistics: the lanes of each codeblock share a subband; two 32x32
    // codeblocks of a warp share it too (warp-uniform)
    bool one_group, same_group;
    // stripe state: significance, signs and their outer neighbours, significant
    // at the plane's start, pending for CP, the plane's bits
    uint32_t S[NQ], N[NQ], H[NQ], HN[NQ], R[NQ], C[NQ], B[NQ];
    // the pass: coded, newly significant (and outer neighbours)
    uint32_t K[NQ], NS[NQ], HNS[NQ];

    BPC_FI Coder(W &w_, const Params &p_, uint32_t *ring_all, const uint8_t *tab_, const uint8_t *,
                 uint32_t (*planes_)[4], uint8_t *, uint32_t *ev_)
        : w(w_), p(p_), tab(tab_), ev(ev_), planes(planes_) {
        evmask = ring_all;
        pfx = ring_all + 256;
        lane = w.lane();
        gl = lane % G::NL;
        const int grp = lane / G::NL;
        gmask = G::NL == 32 ? 0xffffffffu : (0xffffu << (grp * 16));
        ltmask = (1u << lane) - 1u;
        mL = gl > 0 ? EV : 0u;
        mR = gl < G::NL - 1 ? OD : 0u;
    }

    // -------------------------------------------------------------- bit words
    static BPC_FI uint32_t inner(uint32_t x) { return ((x >> 1) & EV) | ((x << 1) & OD); }

    // outer neighbours of x in all words: two words' columns go in one shuffle
    BPC_FI void outer(const uint32_t x[NQ], uint32_t h[NQ]) {
#pragma unroll
        for (int q = 0; q < NQ; q += 2) {
            const uint32_t left = (x[q] & EV) | ((x[q + 1] << 1) & OD), right = ((x[q] >> 1) & EV) | (x[q + 1] & OD);
            const uint32_t a = w.shfl_up(right, 1), b = w.shfl_down(left, 1);
            h[q] = (a & mL) | ((b << 1) & mR);
            h[q + 1] = ((a >> 1) & mL) | (b & mR);
        }
    }

    // full adder: three bits of weight 1 to sum and carry
    static BPC_FI void add3(uint32_t a, uint32_t b, uint32_t c, uint32_t &s, uint32_t &k) {
        s = a ^ b ^ c;
        k = (a & b) | (c & (a ^ b));
    }

    static BPC_FI void rotate(uint32_t a[NQ]) {
        const uint32_t t = a[0];
#pragma unroll
        for (int q = 0; q + 1 < NQ; q++) a[q] = a[q + 1];
        a[NQ - 1] = t;
    }

    // Swap word index bits and the low three bit-index bits of eight words:
    // bit 8i + j of word k becomes bit 8i + k of word j.
    static BPC_FI void transpose8(uint32_t x[8]) {
#pragma unroll
        for (int s = 1; s <= 4; s <<= 1) {
            const uint32_t m = s == 1 ? 0x55555555u : (s == 2 ? 0x33333333u : 0x0F0F0F0Fu);
#pragma unroll
            for (int j = 0; j < 8; j++) {
                if (j & s) continue;
                const uint32_t a = x[j], b = x[j + s];
                x[j] = (a & m) | ((b << s) & ~m);
                x[j + s] = ((a >> s) & m) | (b & ~m);
            }
        }
    }

    // ---------------------------------------------------------------- AC
    // Arithmetic_encoder :261-295 for this lane, with predicated stores
    // instead of branches (lanes reserve at different symbols, and a branch
    // would serialise the warp).  A reservation appends an event: its key, and
    // L, which holds the codeword finished before it.  `on` predicates the
    // call (the optional sign call).
    BPC_FI void symbol(bool on, bool sym, uint32_t P, int key) {
        const bool rs = on && L == E;
        if (rs) put_event(key);
        nev += rs ? 1 : 0;
        L = rs ? 1u : L;
        E = rs ? 0x10000u : E;
        const uint32_t thr = L + (((E - L) * P) >> 7);
        L = on && sym ? thr + 1u : L;
        E = on && !sym ? thr : E;
    }

    BPC_FI void put_event(int key) {
#if defined(__CUDA_ARCH__)
        reinterpret_cast<uint2 *>(ev)[nev] = make_uint2(L, (uint32_t)key);
#else
        ev[2 * nev] = L;
        ev[2 * nev + 1] = (uint32_t)key;
#endif
    }

    BPC_FI void store_open() {
        if (open_slot < 0) return;
        if ((uint32_t)open_slot < (uint32_t)G::CAP)
            slot_out[open_slot] = (int32_t)(L - 1u);
        else
            status |= ST_OVERFLOW;
    }

    // Rank the pass's events by (key, lane); a lane's event e closes the
    // codeword of its event before (or of an earlier pass).
    BPC_FI void rank_events() {
        if (!w.any(nev > 0)) return;
        for (int e = 0; e < nev; e++) w.smem_or(&evmask[ev[2 * e + 1]], 1u << lane);
        w.sync();
        uint32_t c[8], v = 0;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const uint32_t m = evmask[8 * lane + k];
            c[k] = G::NL == 32 ? (uint32_t)popc32(m)
                               : ((uint32_t)popc32(m & 0xFFFFu) | ((uint32_t)popc32(m >> 16) << 16));
            v += c[k];
        }
        const uint32_t own = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = w.shfl_up(v, o);
            if (lane >= o) v += t;
        }
        uint32_t run = v - own;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            pfx[8 * lane + k] = run;
            run += c[k];
        }
        const uint32_t tot = w.shfl_idx(v, 31);
        w.sync();
        const int sh = G::NL == 32 ? 0 : 16 * (lane / G::NL);
        const uint32_t hm = G::NL == 32 ? 0xFFFFFFFFu : 0xFFFFu;
        for (int e = 0; e < nev; e++) {
            const uint32_t key = ev[2 * e + 1];
            const uint32_t slot = 1u + cnt + ((pfx[key] >> sh) & hm) + (uint32_t)popc32(evmask[key] & ltmask & gmask);
            if (open_slot >= 0) {
                if ((uint32_t)open_slot < (uint32_t)G::CAP)
                    slot_out[open_slot] = (int32_t)(ev[2 * e] - 1u);
                else
                    status |= ST_OVERFLOW;
            }
            open_slot = (int)slot;
        }
        cnt += (tot >> sh) & hm;
        nev = 0;
        w.sync();
#pragma unroll
        for (int k = 0; k < 8; k++) evmask[8 * lane + k] = 0u;
        w.sync();
    }

    // ------------------------------------------------------------------ passes
    // 3-pass SPP (:412-456): a non-significant coefficient is coded only if a
    // neighbour is significant when its step comes, and coding can make it
    // significant, so significance spreads within the pass.  Its "dynamic"
    // neighbours are the ones earlier in scan order, so the new significance
    // is the least fixed point of
    //   NS = PN & (static | dyn(NS)),  PN = non-significant with data bit 1,
    // reached from PN & static in as many rounds as the longest chain.
    BPC_FI void spp3(uint32_t am) {
        uint32_t stat[NQ];
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            const uint32_t io = inner(S[q]) | H[q];
            const uint32_t c3 = io | S[q];
            const uint32_t cu = q ? inner(S[q - 1 < 0 ? 0 : q - 1]) | H[q - 1 < 0 ? 0 : q - 1] | S[q - 1 < 0 ? 0 : q - 1] : 0u;
            const uint32_t cd =
                q + 1 < NQ ? inner(S[q + 1 < NQ ? q + 1 : 0]) | H[q + 1 < NQ ? q + 1 : 0] | S[q + 1 < NQ ? q + 1 : 0] : 0u;
            stat[q] = io | (c3 << 2) | (cu >> 30) | (c3 >> 2) | (cd << 30);
            NS[q] = am & ~S[q] & B[q] & stat[q];
        }
        for (;;) {
            bool changed = false;
            outer(NS, HNS);
            uint32_t below = 0u;  // rows 14, 15 of the word above
#pragma unroll
            for (int q = 0; q < NQ; q++) {
                const uint32_t pn = am & ~S[q] & B[q];
                const uint32_t io = inner(NS[q]) | HNS[q], c3 = io | NS[q];
                const uint32_t n = pn & (stat[q] | (c3 << 2) | below | (io & OD));
                below = c3 >> 30;
                changed = changed || n != NS[q];
                NS[q] = n;
            }
            if (!w.any(changed)) break;
        }
        uint32_t below = 0u;
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            const uint32_t io = inner(NS[q]) | HNS[q], c3 = io | NS[q];
            const uint32_t cand = am & ~S[q];
            K[q] = cand & (stat[q] | (c3 << 2) | below | (io & OD));
            below = c3 >> 30;
            C[q] = (C[q] & ~am) | (cand & ~K[q]);  // deferred to CP (:450-452)
        }
    }

    template <int PK>
    BPC_FI void masks(uint32_t am) {
        if constexpr (PK == PK_SPP && PASSES == 3) {
            spp3(am);
        } else {
#pragma unroll
            for (int q = 0; q < NQ; q++) {
                K[q] = am & (PK == PK_CP ? C[q] : ~S[q]);
                NS[q] = K[q] & B[q];
            }
            outer(NS, HNS);
        }
    }

    // The slices of word 0 (the rotated arrays' current word): neighbour count
    // (Compute_Context :164-172) in x[0..3], symbol x[4], sign-context LUT index
    // x[5], x[6] and sign symbol x[7].  Per row, the sum and carry of the three
    // columns around a coefficient serve the rows above and below: above[] =
    // sum and carry (with this pass's significance), significance and signs of
    // the word above (its last row is used), here[] = sum and carry of this
    // word at the pass's start; both are replaced for the next word.
    BPC_FI void slices(int q, uint32_t above[4], uint32_t here[2], uint32_t x[8]) {
        constexpr int nx = NQ > 1 ? 1 : 0;
        const bool last = q == NQ - 1;
        const uint32_t s = S[0], e = s | NS[0], h = H[0], he = h | HNS[0], n = N[0];
        const uint32_t sn = last ? 0u : S[nx], hn_ = last ? 0u : H[nx], nn = last ? 0u : N[nx];
        const uint32_t is = inner(s), ie = inner(e);
        uint32_t su, cu, sd, cd;  // columns of this word as the row below sees them; of the next word
        add3(e, ie, he, su, cu);
        add3(sn, inner(sn), hn_, sd, cd);
        const uint32_t im = (is & EV) | (ie & OD), om = (h & EV) | (he & OD);
        const uint32_t us = (su << 2) | (above[0] >> 30), uc = (cu << 2) | (above[1] >> 30);
        const uint32_t ds = (here[0] >> 2) | (sd << 30), dc = (here[1] >> 2) | (cd << 30);
        uint32_t a, k1, b, k2, k3;
        add3(us, ds, im, a, k1);
        x[0] = a ^ om;
        k2 = a & om;
        add3(uc, dc, k1, b, k3);
        x[1] = b ^ k2;
        k2 = b & k2;
        x[2] = k3 ^ k2;
        x[3] = k3 & k2;
        x[4] = NS[0];
        // Compute_Sign_Context :178-226: with p/m the significant positive /
        // negative neighbours the sums h and v reduce to the classes > 0 and
        // < 0, and the table of :184-208 to three boolean functions of them
        const uint32_t in = inner(n), on = HN[0];
        const uint32_t eu = (e << 2) | (above[2] >> 30), nu = (n << 2) | (above[3] >> 30);
        const uint32_t sb = (s >> 2) | (sn << 30), nb = (n >> 2) | (nn << 30);
        const uint32_t pi = im & ~in, mi = im & in, po = om & ~on, mo = om & on;
        const uint32_t pu = eu & ~nu, mu = eu & nu, pb = sb & ~nb, mb = sb & nb;
        const uint32_t hp = (pi & ~mo) | (po & ~mi), hm = (mi & ~po) | (mo & ~pi);
        const uint32_t vp = (pu & ~mb) | (pb & ~mu), vm = (mu & ~pb) | (mb & ~pu);
        x[5] = (~(hp | hm) & (vp | vm)) | (hp & vp) | (hm & vm);
        x[6] = (hp & ~vm) | (hm & ~vp);
        x[7] = n ^ (hm | (vm & ~hp));
        above[0] = su, above[1] = cu, above[2] = e, above[3] = n;
        here[0] = sd, here[1] = cd;
    }

    // The position at bit f of the bit-reversed K word: its descriptor byte.
    // Word j of the transposed slices is at pfx[32 j + lane], byte i of it the
    // position 8i + j = 31 - f, so i = 3 - f / 8 and j = 7 - f % 8.
    BPC_FI uint32_t descriptor(uint32_t f) const {
        const uint32_t a = (((f * 1025u) >> 3) & 0x383u) ^ (0x383u | ((uint32_t)lane << 2));
        return reinterpret_cast<const uint8_t *>(pfx)[a];
    }

    // the lane's coded symbols of word q (rotated arrays): significance and,
    // for a 1, sign
    BPC_FI void code_word(int q, const uint32_t x[8], int sig_b, uint32_t P4) {
        uint32_t y[8];
#pragma unroll
        for (int k = 0; k < 8; k++) y[k] = x[k];
        transpose8(y);
#pragma unroll
        for (int k = 0; k < 8; k++) pfx[32 * k + lane] = y[k];
        uint32_t k = brev32(K[0]);
        // the next position's descriptor and probability are read ahead of the
        // coder's update for this one (after the last position the reads are
        // of no use, and in range)
        uint32_t f = 31u - (uint32_t)clz32(k), d = descriptor(f), P = tab[sig_b + (int)(d & 15u)];
        while (k) {
            k ^= 1u << f;
            const uint32_t fn = 31u - (uint32_t)clz32(k), dn = descriptor(fn), Pn = tab[sig_b + (int)(dn & 15u)];
            const int key = 64 * q + 62 - 2 * (int)f;
            const bool one = (d & 16u) != 0u;
            symbol(true, one, P, key);
            const uint32_t P2 = perm8(P4, 0x4440u | ((d >> 5) & 3u));
            symbol(one, (d & 128u) != 0u, P2, key + 1);
            f = fn, d = dn, P = Pn;
        }
    }

    // one pass with contexts: SPP or CP
    template <int PK, bool STATS>
    BPC_FI void ctx_pass(int b, bool act, unsigned long long *st) {
        const uint32_t am = act ? ~0u : 0u;
        const int off = PK == PK_CP ? p.cp_off : 0;
        const int sig_b = off + p.a_sig + (g + b) * 9, sign_b = off + p.a_sign + (g + b) * 4;
        masks<PK>(am);
        uint32_t P4 = 0;
        if (!STATS) {
            const uint8_t *sp = tab + sign_b;
            P4 = (uint32_t)sp[0] | ((uint32_t)sp[1] << 8) | ((uint32_t)sp[2] << 16) | ((uint32_t)sp[3] << 24);
        }
        uint32_t above[4] = {0u, 0u, 0u, 0u}, here[2];
        [[maybe_unused]] uint32_t c[13] = {};
        add3(S[0], inner(S[0]), H[0], here[0], here[1]);
#pragma unroll 1
        for (int q = 0; q < NQ; q++) {
            uint32_t x[8];
            slices(q, above, here, x);
            if (!STATS)
                code_word(q, x, sig_b, P4);
            else if (b < 15)
                stats_word(c, x);
            rotate(S), rotate(N), rotate(H), rotate(HN), rotate(NS), rotate(HNS), rotate(K);
        }
        if (!STATS)
            rank_events();
        else if (b < 15)
            stats_store(st, sig_b, sign_b, c);
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            S[q] |= NS[q];
            H[q] |= HNS[q];
            if (PK == PK_CP) C[q] &= ~K[q];
        }
    }

    template <bool STATS>
    BPC_FI void mrp_pass(int b, bool act, unsigned long long *st) {
        if (STATS) {
            uint32_t n = 0, ones = 0;
#pragma unroll
            for (int q = 0; q < NQ; q++) n += (uint32_t)popc32(R[q]), ones += (uint32_t)popc32(R[q] & B[q]);
            if (b >= 15) return;
            if (!act) n = ones = 0;
            uint32_t v = n | (ones << 16);
            if (one_group) {
                v = sum_lanes(v);
                if (gl != 0) v = 0;
            }
            tally(st, g + b, v & 0xFFFFu, v >> 16);
            return;
        }
        const uint32_t P = tab[g + b];
#pragma unroll 1
        for (int q = 0; q < NQ; q++) {
            uint32_t k = act ? brev32(R[0]) : 0u;
            const uint32_t y = brev32(B[0]);
            while (k) {
                const uint32_t f = 31u - (uint32_t)clz32(k), bit = 1u << f;
                k ^= bit;
                symbol(true, (y & bit) != 0u, P, 64 * q + 62 - 2 * (int)f);
            }
            rotate(R), rotate(B);
        }
        rank_events();
    }

    // LUT training (no counterpart in the reference, whose tables come
    // pre-trained): for every LUT entry the pass uses, the number of symbols
    // coded with it and how many of them were 1, counted bit-parallel from
    // the pass masks.  Planes 0..14 only -- the planes of the LUT files, where
    // each entry belongs to exactly one (level, subband, plane, context).
    BPC_FI void tally(unsigned long long *st, int idx, uint32_t n, uint32_t ones) {
        if (n) add_u64(st + 2 * idx, n);
        if (ones) add_u64(st + 2 * idx + 1, ones);
    }
    // A pass's counts, 9 significance contexts and 4 sign ones: symbols in the low
    // half of a word, 1s in the high half (at most 128 a lane, 4096 a codeblock).
    // Atomics are what bounds this kernel, so the counts are summed over the
    // stripe's words and, where the codeblock lies in one subband, over its
    // lanes before they go to memory (4096x4096, 2 passes, 64x64: per word and
    // lane 1545 us, per lane 529, per codeblock 77).
    BPC_FI void stats_word(uint32_t c[13], const uint32_t x[8]) {
#pragma unroll
        for (int k = 0; k < 9; k++) {
            uint32_t m = K[0];
#pragma unroll
            for (int i = 0; i < 4; i++) m &= ((k >> i) & 1) ? x[i] : ~x[i];
            c[k] += (uint32_t)popc32(m) | ((uint32_t)popc32(m & NS[0]) << 16);
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint32_t m = NS[0] & ((k & 1) ? x[5] : ~x[5]) & ((k & 2) ? x[6] : ~x[6]);
            c[9 + k] += (uint32_t)popc32(m) | ((uint32_t)popc32(m & x[7]) << 16);
        }
    }
    BPC_FI uint32_t sum_lanes(uint32_t v) {
#pragma unroll
        for (int o = G::NL / 2; o; o >>= 1) v += w.shfl_xor(v, o);
        return v;
    }
    BPC_FI void stats_store(unsigned long long *st, int sig_b, int sign_b, const uint32_t c[13]) {
        if (one_group) {
            // The counters a lane keeps are halved at each exchange, so lane S k
            // of the codeblock ends with the sum of counter k after 16 shuffles
            // and not 65, and two 32x32 codeblocks of one subband share their
            // atomics (5 levels, 64x64 and 32x32, 512x512 3 passes 45 / 31 -> 43 /
            // 30 us, 4096x4096 3 passes 93 / 84 -> 82 / 73, 2 passes 60 / 72 -> 54 / 50).
            constexpr int S = G::NL / 16;
            uint32_t v[16];
#pragma unroll
            for (int k = 0; k < 16; k++) v[k] = k < 13 ? c[k < 13 ? k : 0] : 0u;
#pragma unroll
            for (int h = 8; h; h >>= 1) {
                const bool up = (gl & (h * S)) != 0;
#pragma unroll
                for (int i = 0; i < h; i++) {
                    const uint32_t keep = up ? v[i + h] : v[i], send = up ? v[i] : v[i + h];
                    v[i] = keep + w.shfl_xor(send, h * S);
                }
            }
            if (S > 1) v[0] += w.shfl_xor(v[0], 1);
            bool mine = gl % S == 0;
            if (same_group) {  // the warp's two 32x32 codeblocks together
                v[0] += w.shfl_xor(v[0], 16);
                mine = lane < 16;
            }
            const int k = gl / S;
            if (mine && k < 13) tally(st, k < 9 ? sig_b + k : sign_b + k - 9, v[0] & 0xFFFFu, v[0] >> 16);
        } else {
#pragma unroll
            for (int k = 0; k < 13; k++) tally(st, k < 9 ? sig_b + k : sign_b + k - 9, c[k] & 0xFFFFu, c[k] >> 16);
        }
    }

    // All-zero codeblock (MSB 32, :1155): 33 planes in which every coefficient
    // is coded with context 0, by SPP (2 passes) or CP (3 passes; SPP defers
    // them all).  The symbols are 0, except in CP at plane 29, where the
    // reference's data bit is its own CP flag (:523-530; the other flag bits
    // read 0 or are never coded here).  Magnitudes out of range (MSB 28..31,
    // flagged) code the same way from their plane down.  All lanes code the
    // same positions, so the warp goes in lockstep, as the decoder does, eight
    // zeros at a time: the lanes' codewords end at the same symbol as a rule
    // (they differ in a codeblock that straddles subbands).  139 -> 109 us
    // for four of them against groups that a spent codeword ended.
    BPC_FI void zero_reserve(bool need) {
        const uint32_t ball = w.ballot(need) & gmask;
        if (need) {
            store_open();
            open_slot = (int)(1u + cnt + (uint32_t)popc32(ball & ltmask));
            L = 1u;
            E = 0x10000u;
        }
        cnt += (uint32_t)popc32(ball);
    }
    BPC_FI void zero_block(bool flat) {
#pragma unroll 1
        for (int b = 32; b >= 0; b--) {
            const bool act = flat && b <= msb;
            const uint32_t P = tab[(PASSES == 3 ? p.cp_off : 0) + p.a_sig + (g + b) * 9];
            const bool one = PASSES == 3 && b == 29;
            // (a probability of 128 or more lets E - L grow)
            const bool runs = !one && P < 128u;
#pragma unroll 1
            for (int t = 0; t < 2 * CBS; t += 8) {
                zero_reserve(act && L == E);
                uint32_t sz = E - L, prev;
                zero_run(sz, prev, P);
                if (!w.any(act && !(runs && prev != 0u))) {
                    if (act) E = L + sz;
                    continue;
                }
                const int n = zero_count(E - L, P);
                uint32_t sz2 = 0xFFFFu;
                bool full = true;
#pragma unroll
                for (int k = 1; k < 8; k++) {
                    if (k < n) continue;
                    full = full && sz2 != 0u;
                    sz2 = (sz2 * P) >> 7;
                }
                const bool same = n == (int)w.shfl_idx((uint32_t)n, lane & ~(G::NL - 1));
                if (!w.any(act && !(runs && n < 8 && same && full))) {
                    zero_reserve(act);
                    if (act) E = L + sz2;
                    continue;
                }
#pragma unroll 1
                for (int k = 0; k < 8; k++) {
                    zero_reserve(act && L == E);
                    const uint32_t thr = L + (((E - L) * P) >> 7);
                    if (act && one) L = thr + 1u;
                    if (act && !one) E = thr;
                }
            }
        }
    }

    // Read_Coefficients :14-44 + Find_MSB :114-161 in one read: per word (16
    // rows of both columns, one 8-byte load a row) the signs go to N, the
    // magnitudes through a bit transpose to bitplanes 0..27 (those up to the
    // word's own highest set bit are stored).  Returns the OR of the magnitudes.
    BPC_FI uint32_t load_planes(const int32_t *src) {
        uint32_t mx = 0;
        qtop = 0u;
#pragma unroll 1
        for (int q = 0; q < NQ; q++) {
            uint32_t a[32], o = 0, n = 0;
#pragma unroll
            for (int r = 0; r < 16; r++) {
                int32_t v0, v1;
                w.load2(src + (size_t)(q * 16 + r) * (size_t)p.X, v0, v1);
                a[2 * r] = v0 < 0 ? 0u - (uint32_t)v0 : (uint32_t)v0;
                a[2 * r + 1] = v1 < 0 ? 0u - (uint32_t)v1 : (uint32_t)v1;
                n |= (uint32_t)(v0 < 0) << (2 * r) | (uint32_t)(v1 < 0) << (2 * r + 1);
                o |= a[2 * r] | a[2 * r + 1];
            }
            mx |= o;
            const int t = o ? 31 - clz32(o) : -1;
            qtop |= (uint32_t)(t + 1) << (8 * q);
            transpose32(a);
#pragma unroll
            for (int k = 0; k < 28; k++)
                if (k <= t) planes[k][q] = a[k];
            N[0] = n;
            rotate(N);
        }
        return mx;
    }

    // ------------------------------------------------------ codeblock driver
    // STATS: gather LUT training counts into `stats` instead of writing the
    // slot stream.
    template <bool STATS = false>
    BPC_FI void run(int cb_first, unsigned long long *stats = nullptr) {
        const int grp = lane / G::NL;
        const int cb = cb_first + grp;
        const bool ok = cb < p.cb_end;
        const int cbx = ok ? cb % p.ncbx : 0, cby = ok ? cb / p.ncbx : 0;
        const int x = cbx * CBS + 2 * gl, y0 = cby * CBS;
        g = lut_group(p, x, y0);
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            S[q] = N[q] = H[q] = HN[q] = 0u;
            C[q] = ~0u;  // CP flag at start (:34-39, :73-78)
        }
        if (STATS) {
            one_group = !w.any(g != (int)w.shfl_idx((uint32_t)g, lane & ~(G::NL - 1)));
            same_group = G::NG > 1 && one_group && !w.any(g != (int)w.shfl_idx((uint32_t)g, 0));
        }
        L = E = 0u;
        cnt = 0u;
        status = 0;
        open_slot = -1;
        nev = 0;
        if (!STATS) {
#pragma unroll
            for (int k = 0; k < 8; k++) evmask[8 * lane + k] = 0u;
            w.sync();
        }
        msb = -1;
        top = -1;
        qtop = 0u;
        slot_out = p.out + (ok ? (size_t)cb * (size_t)G::CAP : 0);
        uint32_t mx = 0;
        if (ok) mx = load_planes(p.in + (size_t)y0 * (size_t)p.X + (size_t)x);
        if (mx >= (1u << 28)) status |= ST_INPUT_RANGE;
#pragma unroll
        for (int o = G::NL / 2; o; o >>= 1) mx |= w.shfl_xor(mx, o);
        if (ok) {
            msb = mx ? 31 - clz32(mx) : 32;
            if (gl == 0 && !STATS) slot_out[0] = msb;  // :1155
            top = msb <= 27 ? msb : -1;  // planes >= 28 are flag bits, not magnitudes
        }
        outer(N, HN);
        const bool flat = msb >= 28;
        if (!STATS && w.any(flat)) zero_block(flat);
        // planes, aligned across the codeblocks that share the warp (LUT
        // training has no entries above plane 14)
        int bmax = flat ? (STATS ? 14 : -1) : msb;
        const int own = bmax;
        if (G::NG > 1) {
            const int other = (int)w.shfl_xor((uint32_t)bmax, 16);
            bmax = other > bmax ? other : bmax;
        }
#pragma unroll 1
        for (int b = bmax; b >= 0; b--) {
            // 2-pass: planes MSB..0 run SPP, MRP.  3-pass: plane MSB runs CP
            // only, planes below run SPP, MRP, CP (:986-1018).
            const bool full = PASSES == 2 ? b <= own : (b < own || (flat && b <= own));
            const bool first_cp = PASSES == 3 && b == own;
#pragma unroll
            for (int q = 0; q < NQ; q++) {
                // a word's planes above its own highest set bit were never
                // stored: they read as zero
                B[q] = b <= top && (uint32_t)b < ((qtop >> (8 * q)) & 0xFFu) ? planes[b][q] : 0u;
                R[q] = S[q];
            }
            if (w.any(full)) {
                ctx_pass<PK_SPP, STATS>(b, full, stats);
                mrp_pass<STATS>(b, full, stats);
            }
            if (PASSES == 3) ctx_pass<PK_CP, STATS>(b, full || first_cp, stats);
        }
        if (ok && !STATS) {
            store_open();  // flush :1020, and the codeword finished last
            // the rest of the slot keeps the -1 fill of :1284
            for (uint32_t k = cnt + 1u + (uint32_t)gl; k < (uint32_t)G::CAP; k += G::NL) slot_out[k] = -1;
            if (cnt + 1u > (uint32_t)G::CAP) status |= ST_OVERFLOW;
        }
        if (ok && p.counts && gl == 0) p.counts[cb] = (int)cnt;
        int st = status;
#pragma unroll
        for (int o = 16; o; o >>= 1) st |= (int)w.shfl_xor((uint32_t)st, o);
        if (st && lane == 0 && p.status) w.atomic_or(p.status, st);
    }
};

}  // namespace bpc
