// bpc_dec.cuh -- the BPC-PaCo codeblock decoder (included by bpc_core.cuh).
//
// What bounds it: integer issue and, for an image of a wave or two, the serial
// chain of the heaviest codeblocks.  A context depends on what the neighbour
// lanes decoded one step earlier, and a reservation needs the number of
// reservations before it, so the warp walks the rows with all lanes together,
// left column then right column, and the work is to make that step short.
//
// State.  Every lane keeps one byte per row of its stripe, four rows to a
// 32-bit word in shared memory ([row / 4][lane], conflict-free):
//   bit 0..3  significance of lane-1's right column, own left, own right,
//             lane+1's left column
//   bit 4..7  their signs (1 = negative; only significant coefficients)
// While a pass walks rows 4g..4g+3 the bytes of rows 4g-1..4g+6 lie in a
// 64-bit register window that moves down one byte per row, so the three rows
// around the current one are always bytes 0..2: every neighbour, the
// coefficient's own bit and every update is a constant mask, the context is
// one AND and one popcount, and the sign context one AND, one multiply (a
// perfect hash of the eight neighbour bits) and one table read.  The right
// column's masks are the left column's shifted by one bit.
//
// Against column masks with variable shifts and per-column halves (B200, same
// launches): 16384x16384 3-pass decode 8.61 -> 4.84 ms, 4096x4096 0.57-1.27 ->
// 0.39 ms (the slow end: images whose clipped areas give all-zero codeblocks,
// 33 planes each, now decoded eight symbols at a time), 2048x2048 2-pass 0.317
// -> 0.241 ms.
#pragma once

namespace bpc {

template <int PASSES, int CBS, class W, int LAT>
struct Coder<PASSES, CBS, false, W, LAT> {
    using G = Geo<CBS>;
    W &w;
    const Params &p;
    const uint8_t *tab;     // LUT bytes
    const uint16_t *sgtab;  // sign-context table (build_sign_table)
    uint32_t *ring;         // codeword window of this lane group's codeblock
    uint32_t *rowbase;      // row words of the warp, [row / 4][lane]
    uint32_t *rows;         // ... this lane's first one
    uint8_t *vis;           // 3 passes: own coefficients SPP coded in the plane, 2 bits a row, [row / 4][lane]
    uint32_t *ref;          // own coefficients significant at the plane's start, [row / 16][lane], bit 2r + c
    // decoded bitplanes, [plane][row / 16]: bit 2r + c = row 16q + r, column c
    // (a per-thread array owned by the caller)
    uint32_t (*planes)[4];
    const int32_t *slot_in;
    uint32_t in_cap;  // words readable at slot_in (slot size, or the compact length)
    int lane, gl, g, msb, status;
    uint32_t gmask, ltmask;
    uint32_t bit_up, bit_dn;  // ballot bit of lane-1 / lane+1 (0 at the codeblock's edge)
    // arithmetic decoder: the interval [L - 1, E - 1] of the codeword cw; L ==
    // E when the codeword is used up
    uint32_t L, E, cw;
    // codeword window: slot words [first, first + RING), the next codeword at
    // word pos of it (group-uniform)
    uint32_t pos, first;
    bool anysig;       // some coefficient of the warp is significant (warp-uniform)
    int sig_base;      // LUT byte index of the current plane and pass
    uint32_t P4;       // its four sign probabilities, one per byte

    BPC_FI Coder(W &w_, const Params &p_, uint32_t *ring_all, const uint8_t *tab_, const uint8_t *sgtab_,
                 uint32_t (*planes_)[4], uint8_t *, uint32_t *)
        : w(w_), p(p_), tab(tab_), sgtab(reinterpret_cast<const uint16_t *>(sgtab_)), planes(planes_) {
        lane = w.lane();
        gl = lane % G::NL;
        const int grp = lane / G::NL;
        gmask = G::NL == 32 ? 0xffffffffu : (0xffffu << (grp * 16));
        ltmask = (1u << lane) - 1u;
        bit_up = gl > 0 ? 1u << ((lane - 1) & 31) : 0u;
        bit_dn = gl < G::NL - 1 ? 1u << ((lane + 1) & 31) : 0u;
        ring = ring_all + grp * G::RING;
        rowbase = ring_all + G::RING * G::NG;
        rows = rowbase + lane;
        ref = rowbase + G::ROW_WORDS + lane;
        vis = reinterpret_cast<uint8_t *>(rowbase + G::ROW_WORDS + G::REF_WORDS) + lane;
    }

    // ---------------------------------------------------------------- AC
    // Lanes with an empty codeword take the next ones in lane order (:268-279);
    // past the slot the window holds the -1 fill (the overflow itself is
    // reported once, from the final count, at the codeblock's end).
    BPC_FI void reserve(bool need, uint32_t ball) {
        const uint32_t bal = ball & gmask;
        if (need) {
            cw = ring[pos + (uint32_t)popc32(bal & ltmask)];
            L = 1u;
            E = 0x10000u;
        }
        pos += (uint32_t)popc32(bal);
    }

    // Arithmetic_decoder :297-339.  With Lower = L - 1 and Size = E - L the
    // reference's Lower + (Size * P >> 7) + 1 is the threshold below, and both
    // outcomes move one end of the interval to it.
    BPC_FI bool ac_step(bool act, uint32_t P) {
        const uint32_t thr = L + (((E - L) * P) >> 7);
        const bool sym = cw >= thr;
        if (act && sym) L = thr + 1u;
        if (act && !sym) E = thr;
        return act && sym;
    }
    template <bool ALWAYS = false>  // reserve without a branch (that nobody reserves is rare)
    BPC_FI bool ac_dec(bool act, uint32_t P) {
        const bool need = act && L == E;
        const uint32_t ball = w.ballot(need);
        if (ALWAYS || ball) reserve(need, ball);  // warp-uniform
        return ac_step(act, P);
    }

    // The codeword window: RING words of the slot from word `first` on, the
    // next codeword at ring[pos].  Before CALLS coder calls (at most NL
    // codewords each): once fewer words are left than those may take, the
    // used ones are dropped and the window is filled up again.
    template <int CALLS>
    BPC_FI void ring_ensure() {
        static_assert(CALLS * G::NL <= G::CHUNK, "");
        if (pos > (uint32_t)(G::RING - CALLS * G::NL)) {  // group-uniform
            w.syncmask(gmask);
            ring_fill<CBS>(ring, slot_in, in_cap, p.offsets != nullptr, first + (uint32_t)G::CHUNK, gl);
            pos -= (uint32_t)G::CHUNK;
            first += (uint32_t)G::CHUNK;
            w.syncmask(gmask);
        }
    }

    // Decoder reconstruction: the reference ORs a plane mask 3 << b into the
    // coefficient (:1038-1083); every bit it sets is later replaced by the
    // decoded bit, so the output holds exactly the decoded bits -- except for
    // MSB = 32, where 3 << 32 is 0 and the mask stays 0 until plane 0 (only
    // plane 0 is read back then).

    // ------------------------------------------------------------- contexts
    template <int CC>
    BPC_FI uint32_t sig_prob(uint32_t lo) const {
        return tab[sig_base + popc32(lo & (kCtxBits << CC))];
    }
    // Compute_Sign_Context :178-226 over left, right, up and below
    template <int CC>
    BPC_FI uint32_t sign_entry(uint32_t lo) const {
        return sgtab[((lo & (kSignBits << CC)) * (kSignHash >> CC)) >> 24];
    }

    // One step: the coefficient of column CC in the row at byte 1 of lo.
    // k8: CP, the row's coefficients SPP coded, at their own bits of lo (9, 10);
    // SPP, collects them at bits 8, 9.
    template <int PK, int CC>
    BPC_FI bool coded_here(uint32_t win, uint32_t &k8, bool act) {
        bool coded = act && ((PK == PK_CP ? win | k8 : win) & (0x200u << CC)) == 0u;
        if (PK == PK_SPP && PASSES == 3) {
            coded = coded && (win & (kCtxBits << CC)) != 0u;  // else it defers to CP (:450-452)
            if (coded) k8 |= 0x100u << CC;
        }
        return coded;
    }
    // the coefficients that became significant (ns, and their ballot) in this
    // lane's byte; the neighbour lane's copy follows from the ballot
    template <int CC>
    BPC_FI void mark(uint32_t &win, bool ns, uint32_t nsb, int shift) {
        if (ns) win |= (0x200u << CC) << shift;
        if (nsb & (CC ? bit_up : bit_dn)) win |= (CC ? 0x100u : 0x800u) << shift;
    }

    template <int PK, int CC>
    BPC_FI void step(uint32_t &lo, uint32_t &k8, bool act) {
        const bool coded = coded_here<PK, CC>(lo, k8, act);
        if (PK == PK_CP || PASSES == 3) {
            if (!w.any(coded)) return;
        }
        const bool ns = ac_dec(coded, sig_prob<CC>(lo));
        const uint32_t nsb = w.ballot(ns);
        if (!nsb) return;
        const uint32_t sg = sign_entry<CC>(lo);
        const bool one = ac_dec(ns, perm8(P4, sg));
        const bool neg = ns && one != ((sg >> 15) != 0u);
        const uint32_t negb = w.ballot(neg);
        mark<CC>(lo, ns, nsb, 0);
        mark<CC>(lo, neg, negb, 4);
    }

    // The latency form.  On an SM with little else to run an ALU operation
    // takes 5 cycles, a compare and a select on it 19, a compare, a vote and a
    // branch on that 46, so the votes are taken in pairs, the sign context is
    // read before the decision, and cx, a copy of lo whose significance bits
    // are complete before the sign call, keeps the next step's context from
    // waiting for this one's signs (one LL codeblock alone, 3 passes: 261 ->
    // 256 us; with MRP reserving without a branch 250 us).
    template <int PK, int CC>
    BPC_FI void step_lat(uint32_t &lo, uint32_t &cx, uint32_t &k8, bool act) {
        const bool coded = coded_here<PK, CC>(cx, k8, act);
        bool need = coded && L == E;
        uint32_t ball = w.ballot(need);
        if (PK == PK_CP || PASSES == 3) {
            if (!w.any(coded)) return;
        }
        const uint32_t sg = sign_entry<CC>(lo);
        if (ball) reserve(need, ball);
        const bool ns = ac_step(coded, sig_prob<CC>(cx));
        const uint32_t nsb = w.ballot(ns);
        need = ns && L == E;
        ball = w.ballot(need);
        if (!nsb) return;
        mark<CC>(cx, ns, nsb, 0);
        if (ball) reserve(need, ball);
        const bool one = ac_step(ns, perm8(P4, sg));
        const bool neg = ns && one != ((sg >> 15) != 0u);
        const uint32_t negb = w.ballot(neg);
        mark<CC>(lo, ns, nsb, 0);
        mark<CC>(lo, neg, negb, 4);
    }

    // Four rows (eight steps) of a codeblock in which nothing is significant
    // yet: every coefficient is coded with context 0, and while all symbols
    // are 0 only E moves, down the same chain whatever the codeword, so one
    // compare against the last threshold decides all eight (zero_run).  The
    // lanes of a codeblock then use up their codewords at the same symbol as a
    // rule, and the next ones, in lane order, are read ahead and tried for the
    // rest of the eight.  False, with at most the first step's reservation
    // made, if a lane decodes a 1 or the lanes differ.  An all-zero codeblock
    // (33 planes, :1155) is decoded entirely here: about 190 -> 44 us, 2
    // passes, against groups that a spent codeword ended.
    BPC_FI bool flat_rows(uint32_t P, bool act) {
        ring_ensure<2>();
        const bool need = act && L == E;
        const uint32_t ball = w.ballot(need);
        if (ball) reserve(need, ball);
        // (probabilities are below 128 in any real table; with others E - L can grow)
        bool ok = P < 128u && E >= L;
        uint32_t sz = E - L, prev;
        zero_run(sz, prev, P);
        if (!w.any(act && !(ok && prev != 0u && cw < L + sz))) {
            if (act) E = L + sz;
            return true;
        }
        const int n = zero_count(E - L, P);
        const uint32_t cw2 = ring[pos + (uint32_t)gl];
        uint32_t sz2 = 0xFFFFu;
        bool full = true;
#pragma unroll
        for (int k = 1; k < 8; k++) {
            if (k < n) continue;
            full = full && sz2 != 0u;
            sz2 = (sz2 * P) >> 7;
        }
        const bool same = n == (int)w.shfl_idx((uint32_t)n, lane & ~(G::NL - 1));
        ok = ok && same && n < 8 && cw < L && full && cw2 < 1u + sz2;
        if (w.any(act && !ok)) return false;
        if (act) {
            cw = cw2;
            L = 1u;
            E = 1u + sz2;
            pos += (uint32_t)G::NL;
        }
        return true;
    }

    // Planes 28..32 of an all-zero codeblock: a symbol cannot make a
    // coefficient significant there (its data bit is one of the reference's
    // flag bits, :523-530), so every one is coded with context 0.
    BPC_FI void high_plane(uint32_t P, bool act) {
#pragma unroll 1
        for (int t = 0; t < 2 * CBS; t += 8) {
            if (flat_rows(P, act)) continue;
#pragma unroll 1
            for (int k = 0; k < 8; k++) {
                ring_ensure<1>();
                (void)ac_dec(act, P);
            }
        }
    }

    template <int PK>
    BPC_FI void ctx_pass(int b, bool act_) {
        // one codeblock a warp: it is active whenever the pass is run
        const bool act = G::NG == 1 || act_;
        const int off = PK == PK_CP ? p.cp_off : 0;
        sig_base = off + p.a_sig + (g + b) * 9;
        const uint8_t *sp = tab + (off + p.a_sign + (g + b) * 4);
        P4 = (uint32_t)sp[0] | ((uint32_t)sp[1] << 8) | ((uint32_t)sp[2] << 16) | ((uint32_t)sp[3] << 24);
        if (PK == PK_SPP && PASSES == 3 && !anysig) return;  // every coefficient defers
        const uint32_t P0 = tab[sig_base];
        if (b > 27) {
            high_plane(P0, act);
            return;
        }
        uint32_t cur = rows[0], last = 0u;
#pragma unroll 1
        for (int q = 0; q < CBS / 4; q++) {
            const uint32_t nxt = q + 1 < CBS / 4 ? rows[(q + 1) * 32] : 0u;
            if (!anysig && (PK == PK_CP || PASSES == 2)) {
                if (flat_rows(P0, act)) continue;
            }
            uint32_t lo = (cur << 8) | last, hi = (cur >> 24) | (nxt << 8), out = 0u;
            [[maybe_unused]] uint32_t cx = lo;
            uint32_t k8 = PASSES == 3 && PK == PK_CP ? (uint32_t)vis[q * 32] << 9 : 0u;
#pragma unroll 1
            for (int r = 0; r < 4; r++) {
                ring_ensure<4>();  // two steps of up to two calls
                if constexpr (LAT > 0) {
                    step_lat<PK, 0>(lo, cx, k8, act);
                    step_lat<PK, 1>(lo, cx, k8, act);
                    cx = funnel_r(cx, hi, 8);
                } else {
                    step<PK, 0>(lo, k8, act);
                    step<PK, 1>(lo, k8, act);
                }
                lo = funnel_r(lo, hi, 8);
                hi >>= 8;
                out = (out >> 8) | (lo << 24);
                k8 >>= 2;
            }
            rows[q * 32] = out;
            if (!anysig) anysig = w.any(out != 0u);
            if (PASSES == 3 && PK == PK_SPP) vis[q * 32] = (uint8_t)k8;
            last = out >> 24;
            cur = nxt;
        }
    }

    // own bits (bit s and s + 1 of each row byte) of 16 rows, as bit 2r + c
    BPC_FI uint32_t own16(int q, int s) const {
        uint32_t v = 0;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint32_t x = (rows[(4 * q + k) * 32] >> s) & 0x03030303u;
            v = (v >> 8) | ((x * 0x01041040u) & 0xff000000u);
        }
        return v;
    }

    // MRP_Decoder :608-629 over the coefficients significant at the plane's
    // start; only the steps where some lane has one are run.  (Letting each
    // lane decode on its own until its codeword is used up, and ranking the
    // waiting lanes by position, needs fewer votes but measured slower on the
    // serial chain of one codeblock: 187 -> 202 us, 2 passes.)
    BPC_FI void mrp_pass(int b, bool act) {
        if (b > 27) return;  // nothing can be significant
        const uint32_t P = tab[g + b];
#pragma unroll 1
        for (int q = 0; q < CBS / 16; q++) {
            const uint32_t R = G::NG == 1 || act ? ref[q * 32] : 0u;
            uint32_t bits = 0;
            uint32_t u = anysig ? w.reduce_or(R) : 0u;
            while (u) {
                const uint32_t bit = u & (0u - u);
                u ^= bit;
                ring_ensure<1>();
                if (ac_dec<(LAT > 0)>((R & bit) != 0u, P)) bits |= bit;
            }
            planes[b][q] = bits;
        }
    }

    // the plane's newly significant coefficients are 1-bits too; what is
    // significant now is refined in the next plane
    BPC_FI void plane_end(int b, bool mrp) {
        if (b > 27) return;
        if (!anysig) {
#pragma unroll
            for (int q = 0; q < CBS / 16; q++) planes[b][q] = 0u;
            return;
        }
#pragma unroll 1
        for (int q = 0; q < CBS / 16; q++) {
            const uint32_t sg = own16(q, 1), r = ref[q * 32];
            planes[b][q] = (mrp ? planes[b][q] : 0u) | (sg & ~r);
            ref[q * 32] = sg;
        }
    }

    // Write_Coefficients :46-63: planes back to magnitudes, 16 rows of both
    // columns at a time; a row's two coefficients go out in one 8-byte store
    // where the raster is 8-byte aligned
    BPC_FI void write_rows(int32_t *dst, bool vec, const uint32_t a[32], uint32_t neg) {
#pragma unroll
        for (int r = 0; r < 16; r++) {
            const uint32_t s0 = 0u - ((neg >> (2 * r)) & 1u), s1 = 0u - ((neg >> (2 * r + 1)) & 1u);
            const int32_t v0 = (int32_t)((a[2 * r] ^ s0) - s0), v1 = (int32_t)((a[2 * r + 1] ^ s1) - s1);
            int32_t *d = dst + (size_t)r * (size_t)p.X;
            if (vec) {
                w.store2(d, v0, v1);
            } else {
                w.store1(d, v0);
                w.store1(d + 1, v1);
            }
        }
    }

    // ------------------------------------------------------ codeblock driver
    BPC_FI void run(int cb_first) {
        const int grp = lane / G::NL;
        const int cb = cb_first + grp;
        const bool ok = cb < p.cb_end;
        const int cbx = ok ? cb % p.ncbx : 0, cby = ok ? cb / p.ncbx : 0;
        const int x = cbx * CBS + 2 * gl, y0 = cby * CBS;
        g = lut_group(p, x, y0);
        L = E = cw = 0u;
        pos = 1u;
        first = 0u;
        status = 0;
        anysig = false;
        msb = -1;
        const uint32_t cap = (uint32_t)G::CAP;
        if (p.offsets) {  // compact container; words past the codeblock read as the -1 fill
            const long long o0 = ok ? p.offsets[cb] : 0, o1 = ok ? p.offsets[cb + 1] : 0;
            // damaged offsets (outside the container, or decreasing) read
            // nothing: the codeblock then decodes as a bad stream
            const bool inside = o0 >= 0 && o1 >= o0 && o1 <= p.in_words;
            slot_in = p.in + (inside ? o0 : 0);
            const long long n = inside ? o1 - o0 : 0;
            in_cap = (uint32_t)(n > (long long)cap ? (long long)cap : n);
        } else {
            slot_in = p.in + (ok ? (size_t)cb * (size_t)cap : 0);
            in_cap = cap;
        }
        w.sync();  // the last codeblock's reads of the ring are over
        if (ok) {
            ring_fill<CBS>(ring, slot_in, in_cap, p.offsets != nullptr, 0u, gl);
        }
#pragma unroll
        for (int q = 0; q < CBS / 4; q++) {
            rows[q * 32] = 0u;
            if (PASSES == 3) vis[q * 32] = 0;
        }
#pragma unroll
        for (int q = 0; q < CBS / 16; q++) ref[q * 32] = 0u;
        w.sync();
        if (ok) {
            const int m = (int)ring[0];  // :1216
            // an encoder writes 0..27 (|x| < 2^28) or 32 (all-zero block)
            if ((m >= 0 && m <= 27) || m == 32)
                msb = m;
            else
                status |= ST_BAD_STREAM;
        }
        // planes, aligned across the codeblocks that share the warp
        int bmax = msb;
        if (G::NG > 1) {
            const int other = (int)w.shfl_xor((uint32_t)bmax, 16);
            bmax = other > bmax ? other : bmax;
        }
#pragma unroll 1
        for (int b = bmax; b >= 0; b--) {
            // 2-pass: planes MSB..0 run SPP, MRP.  3-pass: plane MSB runs CP
            // only, planes below run SPP, MRP, CP (:986-1018).
            const bool full = PASSES == 2 ? b <= msb : b < msb;
            const bool first_cp = PASSES == 3 && b == msb;
            const bool mrp = w.any(full);
            if (mrp) {
                ctx_pass<PK_SPP>(b, full);
                mrp_pass(b, full);
            }
            if (PASSES == 3) ctx_pass<PK_CP>(b, full || first_cp);
            plane_end(b, mrp);
        }
        // planes 0..top are read back
        const int top = msb == 32 ? 0 : msb;
        if (ok) {
            int32_t *dst = p.out + (size_t)y0 * (size_t)p.X + (size_t)x;
            const bool vec = (((uintptr_t)p.out) & 7u) == 0u;
#pragma unroll 1
            for (int q = 0; q < CBS / 16; q++) {
                uint32_t a[32];
#pragma unroll
                for (int k = 0; k < 32; k++) a[k] = (k < 28 && k <= top) ? planes[k < 28 ? k : 0][q] : 0u;
                transpose32(a);
                write_rows(dst + (size_t)(16 * q) * (size_t)p.X, vec, a, own16(q, 5));
            }
            const uint32_t cnt = first + pos - 1u;  // codewords reserved
            if (cnt >= cap) status |= ST_OVERFLOW;  // a reservation read past the slot
            if (p.counts && gl == 0) p.counts[cb] = (int)cnt;
        }
        int st = status;
        for (int o = 16; o; o >>= 1) st |= (int)w.shfl_xor((uint32_t)st, o);
        if (st && lane == 0 && p.status) w.atomic_or(p.status, st);
    }
};

}  // namespace bpc
