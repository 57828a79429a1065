#pragma once

namespace bpc {

struct Lane {
    uint64_t S[2], R[2], C[2], N[2];
    uint64_t XL, XR, XNL, XNR;
    uint32_t lower, size, resv, cw;
    uint32_t cnt;
    int status;
    int open_slot;
    int cur_ev;
    int nev;
};

template <int PASSES, int CBS, class W, int LAT>
struct Coder<PASSES, CBS, true, W, LAT> {
    using G = Geo<CBS>;
    static constexpr int NH = CBS / 32;  // 32-row halves per column
    W &w;
    const Params &p;
    Lane s;
    const uint8_t *tab;    // LUT bytes
    int32_t *slot_out;
    int lane, gl, g, msb;
    int top;        // highest bitplane coded from the stored planes (-1: none)
    uint32_t qtop;  // encoder: per quarter q, byte q = 1 + the highest plane stored for it (0: none)
    uint32_t gmask, ltmask;
    uint64_t B[2];  // encoder: magnitude bits of the current plane; decoder: decoded 1-bits
    int sig_base, sign_base;  // LUT byte indices of the current plane and pass
    // encoder, per pass: coded (K), symbol-1 (Y) and newly significant (NS)
    // masks, neighbour columns' significance at pass start and new in pass
    uint64_t K[2], Y[2], NS[2], XLS, XRS, XLN, XRN;
    uint64_t cs[2][4];  // context bit slices per column
    uint64_t si[2][2];  // sign-context LUT index bit slices per column
    uint64_t sg[2];     // sign symbol per column (own sign ^ predicted sign)
    uint32_t *evmask;   // per warp, 256 keys: lanes with a reservation event
    uint32_t *pfx;      // per warp, 256 keys: events before the key (ranking)
    uint8_t *ev_key;    // this lane's events of the pass: key, finished codeword
    uint32_t *ev_val;
    // bitplanes, [plane][col0 rows 0-31, col0 rows 32-63, col1 rows 0-31, col1 rows 32-63]
    // (per-thread arrays owned by the caller: an array indexed at run time
    // inside this struct would keep the whole struct out of registers)
    uint32_t (*planes)[4];

    BPC_FI Coder(W &w_, const Params &p_, uint32_t *ring_all, const uint8_t *tab_, const uint8_t *,
                 uint32_t (*planes_)[4], uint8_t *ev_key_, uint32_t *ev_val_)
        : w(w_), p(p_), tab(tab_), planes(planes_), ev_key(ev_key_), ev_val(ev_val_) {
        evmask = ring_all;
        pfx = ring_all + 256;
        lane = w.lane();
        gl = lane % G::NL;
        const int grp = lane / G::NL;
        gmask = G::NL == 32 ? 0xffffffffu : (0xffffu << (grp * 16));
        ltmask = (1u << lane) - 1u;
    }

    // magnitude bits of plane b
    BPC_FI void plane_begin(int b) {
        if (b <= top) {
            // a quarter's planes above its own highest set bit were never
            // stored: they read as zero
            const uint32_t *q = planes[b];
            const uint32_t u = (uint32_t)b;
            const uint32_t q0 = u < (qtop & 0xFFu) ? q[0] : 0u, q1 = u < ((qtop >> 8) & 0xFFu) ? q[1] : 0u;
            const uint32_t q2 = u < ((qtop >> 16) & 0xFFu) ? q[2] : 0u, q3 = u < (qtop >> 24) ? q[3] : 0u;
            B[0] = (uint64_t)q0 | ((uint64_t)q1 << 32);
            B[1] = (uint64_t)q2 | ((uint64_t)q3 << 32);
        } else {
            B[0] = B[1] = 0ull;
        }
    }

    // ---------------------------------------------------- encoder, decoupled
    // The encoder knows every data bit up front, so per pass it computes, for
    // all rows at once, which coefficients are coded (K), which code a 1 (Y),
    // which become significant (NS) and their contexts from time-accurate
    // neighbour significance (earlier in scan order: start of pass | NS; later:
    // start of pass).  Each lane then runs its arithmetic coder over its own
    // coded symbols only.  A reservation (:268-279) is recorded as an event
    // keyed by (row, column, phase) inside a 16-row chunk; after the chunk the
    // warp ranks all events by (key, lane) -- the reference's lockstep order --
    // and the codewords go to their slots.

    // Arithmetic_encoder :261-295 for this lane, with predicated stores
    // instead of branches (lanes reserve and finish codewords at different
    // symbols, and a branch per case would serialise the warp).  A reservation
    // (:268-279) appends an event (its key; the slot is ranked at the end of
    // the pass); a finished codeword (Size == 0) stores its value with its
    // event, or in ev_val[kEvOpen] if it was reserved in an earlier pass.
    // `on` predicates the call (the optional sign call).
    BPC_FI void enc_symbol_if(bool on, uint32_t sym, uint32_t P, int key) {
        const bool rs = on && s.size == 0;
        if (rs) ev_key[s.nev] = (uint8_t)key;
        s.cur_ev = rs ? s.nev : s.cur_ev;
        s.nev += rs ? 1 : 0;
        const uint32_t size0 = rs ? 0xFFFFu : s.size, low0 = rs ? 0u : s.lower;
        const uint32_t t = ((size0 * P) >> 7) + sym;
        const uint32_t nsize = sym ? size0 - t : t;
        const uint32_t nlow = sym ? low0 + t : low0;
        const bool fin = on && nsize == 0;
        if (fin) ev_val[s.cur_ev] = nlow;
        s.size = on ? nsize : s.size;
        s.lower = on ? nlow : s.lower;
    }

    // Rank the pass's events by (key, lane) and store completed codewords.
    BPC_FI void enc_rank() {
        // The codeword left open by an earlier pass finished in this one if the
        // lane reserved again (a reservation needs Size == 0) or ends at Size 0.
        if (s.open_slot >= 0 && (s.nev > 0 || s.size == 0)) {
            if ((uint32_t)s.open_slot < (uint32_t)G::CAP)
                slot_out[s.open_slot] = (int32_t)ev_val[kEvOpen];
            else
                s.status |= ST_OVERFLOW;
            s.open_slot = -1;
        }
        if (!w.any(s.nev > 0)) return;
        for (int e = 0; e < s.nev; e++) w.smem_or(&evmask[ev_key[e]], 1u << lane);
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
        for (int e = 0; e < s.nev; e++) {
            const int key = ev_key[e];
            const uint32_t slot = 1u + s.cnt + ((pfx[key] >> sh) & hm) + (uint32_t)popc32(evmask[key] & ltmask & gmask);
            if (e < s.nev - 1 || s.size == 0) {
                if (slot < (uint32_t)G::CAP)
                    slot_out[slot] = (int32_t)ev_val[e];
                else
                    s.status |= ST_OVERFLOW;
            } else {
                s.open_slot = (int)slot;
            }
        }
        s.cnt += (tot >> sh) & hm;
        s.cur_ev = kEvOpen;  // a codeword still open finishes into ev_val[kEvOpen]
        s.nev = 0;
        w.sync();
#pragma unroll
        for (int k = 0; k < 8; k++) evmask[8 * lane + k] = 0u;
        w.sync();
    }

    // lane-1's new right column and lane+1's new left column
    BPC_FI void enc_neighbour_ns() {
        const uint64_t up = shfl_up64(w, NS[1]), dn = shfl_down64(w, NS[0]);
        XLN = gl > 0 ? up : 0ull;
        XRN = gl < G::NL - 1 ? dn : 0ull;
    }

    // Compute_Context :164-172 for every row, with the neighbours' significance
    // as each coefficient's step sees it (Share_*_Borders :342-388).
    BPC_FI void enc_contexts() {
        const uint64_t S0 = s.S[0], S1 = s.S[1];
        const uint64_t Le = S0 | NS[0], Re = S1 | NS[1], XLe = XLS | XLN, XRe = XRS | XRN;
        uint64_t x[8];
        x[0] = XLe << 1;  // (i-1, lane-1 right)
        x[1] = Le << 1;   // (i-1, left)
        x[2] = Re << 1;   // (i-1, right)
        x[3] = XLS;       // (i, lane-1 right): later in scan
        x[4] = S1;        // (i, right): later
        x[5] = XLS >> 1;  // (i+1, *): later
        x[6] = S0 >> 1;
        x[7] = S1 >> 1;
        count8(x, cs[0][0], cs[0][1], cs[0][2], cs[0][3]);
        x[0] = Le << 1;
        x[1] = Re << 1;
        x[2] = XRe << 1;
        x[3] = Le;   // (i, left): earlier in scan
        x[4] = XRe;  // (i, lane+1 left): earlier
        x[5] = S0 >> 1;
        x[6] = S1 >> 1;
        x[7] = XRS >> 1;
        count8(x, cs[1][0], cs[1][1], cs[1][2], cs[1][3]);
    }

    // Compute_Sign_Context :178-226 for every row at once.  With pos/neg the
    // significant-positive / significant-negative neighbours, the sums
    // h = sgn(l) + sgn(r) and v = sgn(u) + sgn(b) reduce to the classes
    // h > 0 = (pl & ~nr) | (pr & ~nl), h < 0 = (nl & ~pr) | (nr & ~pl), and the
    // table of :184-208 to three boolean functions of the classes: the LUT
    // index (ctx >> 1) bits and the predicted-sign bit (ctx & 1).
    BPC_FI void enc_sign_slices() {
        const uint64_t Le = s.S[0] | NS[0], Re = s.S[1] | NS[1], XRe = XRS | XRN;
#pragma unroll
        for (int c = 0; c < 2; c++) {
            uint64_t sl, nl, sr, nr, su, nu, sb, nb;
            if (c == 0) {
                sl = XLS; nl = s.XNL;                   // (i, lane-1 right): later
                sr = s.S[1]; nr = s.N[1];               // (i, right): later
                su = Le << 1; nu = s.N[0] << 1;         // (i-1, left): earlier
                sb = s.S[0] >> 1; nb = s.N[0] >> 1;     // (i+1, left): later
            } else {
                sl = Le; nl = s.N[0];                   // (i, left): earlier
                sr = XRe; nr = s.XNR;                   // (i, lane+1 left): earlier
                su = Re << 1; nu = s.N[1] << 1;
                sb = s.S[1] >> 1; nb = s.N[1] >> 1;
            }
            const uint64_t pl = sl & ~nl, ml = sl & nl, pr = sr & ~nr, mr = sr & nr;
            const uint64_t pu = su & ~nu, mu = su & nu, pb = sb & ~nb, mb = sb & nb;
            const uint64_t hp = (pl & ~mr) | (pr & ~ml), hn = (ml & ~pr) | (mr & ~pl);
            const uint64_t vp = (pu & ~mb) | (pb & ~mu), vn = (mu & ~pb) | (mb & ~pu);
            const uint64_t h0 = ~(hp | hn), v0 = ~(vp | vn);
            si[c][0] = (h0 & ~v0) | (hp & vp) | (hn & vn);
            si[c][1] = (hp & ~vn) | (hn & ~vp);
            sg[c] = s.N[c] ^ ((h0 & vn) | hn);
        }
    }

    // Compute_Sign_Context :214-226 for a coefficient that became significant
    BPC_FI int enc_sign_ctx(int i, int c) {
        const uint64_t Le = s.S[0] | NS[0], Re = s.S[1] | NS[1];
        // c is a runtime value here: select, never index (keeps the state in registers)
        const uint64_t Me = c ? Re : Le, Ml = c ? s.S[1] : s.S[0], Nc = c ? s.N[1] : s.N[0];
        const int us = i ? (int)bit64(Me, i - 1) : 0, un = i ? (int)bit64(Nc, i - 1) : 0;
        const int bs = (int)bit64(Ml >> 1, i), bn = (int)bit64(Nc >> 1, i);
        int ls, ln, rs, rn;
        if (c == 0) {
            ls = (int)bit64(XLS, i);
            ln = (int)bit64(s.XNL, i);
            rs = (int)bit64(s.S[1], i);
            rn = (int)bit64(s.N[1], i);
        } else {
            ls = (int)bit64(Le, i);
            ln = (int)bit64(s.N[0], i);
            rs = (int)bit64(XRS | XRN, i);
            rn = (int)bit64(s.XNR, i);
        }
        const int h = ls * (1 - 2 * ln) + rs * (1 - 2 * rn);
        const int v = us * (1 - 2 * un) + bs * (1 - 2 * bn);
        const int hc = h == 0 ? 0 : (h > 0 ? 1 : 2), vc = v == 0 ? 0 : (v > 0 ? 1 : 2);
        return (int)((kSignTab >> (3 * (hc * 3 + vc))) & 7u);
    }

    // 3-pass SPP (:412-456): a non-significant coefficient is coded only if a
    // neighbour is significant when its step comes, and coding can make it
    // significant, so significance spreads within the pass.  A coefficient's
    // "dynamic" neighbours are the ones earlier in scan order, so the new
    // significance set is the least fixed point of
    //   new = PN & (static | dyn(new)),  PN = non-significant with data bit 1,
    // reached from new = PN & static in as many rounds as the longest chain.
    BPC_FI void enc_spp3_propagate(bool act, bool lowp) {
        const uint64_t S0 = s.S[0], S1 = s.S[1];
        const uint64_t dXL = XLS | (XLS << 1) | (XLS >> 1), dXR = XRS | (XRS << 1) | (XRS >> 1);
        const uint64_t dS0 = S0 | (S0 << 1) | (S0 >> 1), dS1 = S1 | (S1 << 1) | (S1 >> 1);
        const uint64_t statL = dXL | (S0 << 1) | (S0 >> 1) | dS1;
        const uint64_t statR = dS0 | (S1 << 1) | (S1 >> 1) | dXR;
        const uint64_t cand0 = act ? ~S0 & G::ROWS : 0ull, cand1 = act ? ~S1 & G::ROWS : 0ull;
        const uint64_t pn0 = lowp ? cand0 & B[0] : 0ull, pn1 = lowp ? cand1 & B[1] : 0ull;
        uint64_t ns0 = pn0 & statL, ns1 = pn1 & statR, nxl = 0, nxr = 0;
        for (;;) {
            const uint64_t up = shfl_up64(w, ns1), dn = shfl_down64(w, ns0);
            nxl = gl > 0 ? up : 0ull;
            nxr = gl < G::NL - 1 ? dn : 0ull;
            const uint64_t n0 = pn0 & (statL | ((nxl | ns0 | ns1) << 1));
            const uint64_t n1 = pn1 & (statR | ((n0 | ns1 | nxr) << 1) | n0 | nxr);
            const bool changed = (n0 != ns0) || (n1 != ns1);
            ns0 = n0;
            ns1 = n1;
            if (!w.any(changed)) break;
        }
        NS[0] = ns0;
        NS[1] = ns1;
        XLN = nxl;
        XRN = nxr;
        const uint64_t dynL = (nxl | ns0 | ns1) << 1;
        const uint64_t dynR = ((ns0 | ns1 | nxr) << 1) | ns0 | nxr;
        K[0] = cand0 & (statL | dynL);
        K[1] = cand1 & (statR | dynR);
        s.C[0] |= cand0 & ~K[0];  // deferred to CP (:450-452)
        s.C[1] |= cand1 & ~K[1];
    }

    // One pass = masks (what is coded, with which context and symbol), code
    // (the lane's arithmetic coder over those symbols, events ranked) and
    // commit (the state the next pass sees).  LUT training replaces the code
    // step with stats_pass.
    template <int PK>
    BPC_FI void enc_pass(int b, bool act) {
        enc_pass_masks<PK>(b, act);
        enc_pass_code<PK>(b, act);
        enc_pass_commit<PK>(act);
    }

    template <int PK>
    BPC_FI void enc_pass_masks(int b, bool act) {
        // The data bit coded at plane b is magnitude bit b for b <= 27; above
        // that the reference reads its flag bits (b+1 = 29 refinement, 30 CP,
        // 31 significance, >= 32 nothing), which for the coefficients each pass
        // visits are constants: MRP reads 1 at b = 28 and 30, CP reads 1 at
        // b = 29 (the CP flag itself) without the coefficient becoming
        // significant (:523-530).  Planes >= 28 only occur for MSB 32.
        const bool lowp = b <= 27;
#pragma unroll
        for (int c = 0; c < 2; c++) {
            if (PK == PK_MRP) {
                K[c] = act ? s.R[c] : 0ull;
                Y[c] = lowp ? (K[c] & B[c]) : ((b == 28 || b == 30) ? K[c] : 0ull);
                NS[c] = 0ull;
            } else if (PK == PK_CP) {
                K[c] = act ? s.C[c] : 0ull;
                NS[c] = lowp ? (K[c] & B[c]) : 0ull;
                Y[c] = lowp ? NS[c] : (b == 29 ? K[c] : 0ull);
            } else if (PASSES == 2) {
                K[c] = act ? (~s.S[c] & G::ROWS) : 0ull;
                NS[c] = lowp ? (K[c] & B[c]) : 0ull;
                Y[c] = NS[c];
            }
        }
        if (PK == PK_SPP && PASSES == 3) {
            enc_spp3_propagate(act, lowp);
            Y[0] = NS[0];
            Y[1] = NS[1];
        } else if (PK != PK_MRP) {
            enc_neighbour_ns();
        }
        if (PK != PK_MRP) {
            enc_contexts();
            enc_sign_slices();
        }
    }

    // significance context of position t from its four bit slices
    static BPC_FI uint32_t ctx4(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3, int t) {
        return ((c0 >> t) & 1u) | (((c1 >> t) & 1u) << 1) | (((c2 >> t) & 1u) << 2) | (((c3 >> t) & 1u) << 3);
    }

    template <int PK>
    BPC_FI void enc_pass_code(int b, bool act) {
        const int off = PK == PK_CP ? p.cp_off : 0;
        const int sig_b = off + p.a_sig + (g + b) * 9, sign_b = off + p.a_sign + (g + b) * 4;
        const uint32_t Pref = PK == PK_MRP && act ? (uint32_t)tab[g + b] : 0u;
        // one lane's coded symbols in scan order: 16 rows at a time, the two
        // columns interleaved so that position t = 2*row + column
#pragma unroll 1
        for (int q = 0; q < CBS / 16; q++) {
            uint32_t kq = zip16(K[0], K[1], q);
            if (!kq) continue;
            const uint32_t yq = zip16(Y[0], Y[1], q);
            uint32_t nq = 0, c0 = 0, c1 = 0, c2 = 0, c3 = 0, s0 = 0, s1 = 0, gq = 0;
            if (PK != PK_MRP) {
                nq = zip16(NS[0], NS[1], q);
                c0 = zip16(cs[0][0], cs[1][0], q);
                c1 = zip16(cs[0][1], cs[1][1], q);
                c2 = zip16(cs[0][2], cs[1][2], q);
                c3 = zip16(cs[0][3], cs[1][3], q);
                s0 = zip16(si[0][0], si[1][0], q);
                s1 = zip16(si[0][1], si[1][1], q);
                gq = zip16(sg[0], sg[1], q);
            }
            if constexpr (LAT >= 2) {  // three positions per iteration, the later ones predicated
                do {
                    const int t = ctz32(kq);
                    kq &= kq - 1;
                    const bool two = kq != 0u;
                    const int t2 = two ? ctz32(kq) : t;
                    kq &= two ? kq - 1 : kq;
                    const bool three = kq != 0u;
                    const int t3 = three ? ctz32(kq) : t;
                    kq &= three ? kq - 1 : kq;
                    const int key = (32 * q + t) * 2, key2 = (32 * q + t2) * 2, key3 = (32 * q + t3) * 2;
                    if (PK == PK_MRP) {
                        enc_symbol_if(true, (yq >> t) & 1u, Pref, key);
                        enc_symbol_if(two, (yq >> t2) & 1u, Pref, key2);
                        enc_symbol_if(three, (yq >> t3) & 1u, Pref, key3);
                    } else {
                        const uint32_t ca = ctx4(c0, c1, c2, c3, t), cb2 = ctx4(c0, c1, c2, c3, t2);
                        const uint32_t cc3 = ctx4(c0, c1, c2, c3, t3);
                        const uint32_t sa = ((s0 >> t) & 1u) | (((s1 >> t) & 1u) << 1);
                        const uint32_t sb = ((s0 >> t2) & 1u) | (((s1 >> t2) & 1u) << 1);
                        const uint32_t sc = ((s0 >> t3) & 1u) | (((s1 >> t3) & 1u) << 1);
                        const uint32_t Pa = tab[sig_b + (int)ca], P2a = tab[sign_b + (int)sa];
                        const uint32_t Pb = tab[sig_b + (int)cb2], P2b = tab[sign_b + (int)sb];
                        const uint32_t Pc = tab[sig_b + (int)cc3], P2c = tab[sign_b + (int)sc];
                        enc_symbol_if(true, (yq >> t) & 1u, Pa, key);
                        enc_symbol_if(((nq >> t) & 1u) != 0u, (gq >> t) & 1u, P2a, key + 1);
                        enc_symbol_if(two, (yq >> t2) & 1u, Pb, key2);
                        enc_symbol_if(two && ((nq >> t2) & 1u) != 0u, (gq >> t2) & 1u, P2b, key2 + 1);
                        enc_symbol_if(three, (yq >> t3) & 1u, Pc, key3);
                        enc_symbol_if(three && ((nq >> t3) & 1u) != 0u, (gq >> t3) & 1u, P2c, key3 + 1);
                    }
                } while (kq);
            } else if constexpr (LAT == 1) {  // two positions per iteration, the second predicated
                do {
                    const int t = ctz32(kq);
                    kq &= kq - 1;
                    const bool two = kq != 0u;
                    const int t2 = two ? ctz32(kq) : t;
                    kq &= two ? kq - 1 : kq;
                    const int key = (32 * q + t) * 2, key2 = (32 * q + t2) * 2;
                    if (PK == PK_MRP) {
                        enc_symbol_if(true, (yq >> t) & 1u, Pref, key);
                        enc_symbol_if(two, (yq >> t2) & 1u, Pref, key2);
                    } else {
                        const uint32_t ca = ctx4(c0, c1, c2, c3, t), cb2 = ctx4(c0, c1, c2, c3, t2);
                        const uint32_t sa = ((s0 >> t) & 1u) | (((s1 >> t) & 1u) << 1);
                        const uint32_t sb = ((s0 >> t2) & 1u) | (((s1 >> t2) & 1u) << 1);
                        const uint32_t Pa = tab[sig_b + (int)ca], P2a = tab[sign_b + (int)sa];
                        const uint32_t Pb = tab[sig_b + (int)cb2], P2b = tab[sign_b + (int)sb];
                        enc_symbol_if(true, (yq >> t) & 1u, Pa, key);
                        enc_symbol_if(((nq >> t) & 1u) != 0u, (gq >> t) & 1u, P2a, key + 1);
                        enc_symbol_if(two, (yq >> t2) & 1u, Pb, key2);
                        enc_symbol_if(two && ((nq >> t2) & 1u) != 0u, (gq >> t2) & 1u, P2b, key2 + 1);
                    }
                } while (kq);
            } else {
                do {
                    const int t = ctz32(kq);
                    kq &= kq - 1;
                    const int key = (32 * q + t) * 2;  // (row, column, phase) in the pass
                    if (PK == PK_MRP) {
                        enc_symbol_if(true, (yq >> t) & 1u, Pref, key);
                    } else {
                        const uint32_t ctx = ctx4(c0, c1, c2, c3, t);
                        enc_symbol_if(true, (yq >> t) & 1u, tab[sig_b + (int)ctx], key);
                        // the sign call of a coefficient that became significant
                        const uint32_t sidx = ((s0 >> t) & 1u) | (((s1 >> t) & 1u) << 1);
                        enc_symbol_if(((nq >> t) & 1u) != 0u, (gq >> t) & 1u, tab[sign_b + (int)sidx], key + 1);
                    }
                } while (kq);
            }
        }
        enc_rank();
    }

    template <int PK>
    BPC_FI void enc_pass_commit(bool act) {
        if (PK == PK_MRP) {
            if (act) {
                s.R[0] = s.S[0];
                s.R[1] = s.S[1];
            }
        } else {
            s.S[0] |= NS[0];
            s.S[1] |= NS[1];
            XLS |= XLN;
            XRS |= XRN;
            if (PK == PK_CP) {
                s.R[0] |= NS[0];
                s.R[1] |= NS[1];
                s.C[0] &= ~K[0];
                s.C[1] &= ~K[1];
            }
        }
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
    template <int PK>
    BPC_FI void stats_pass(int b, bool act, unsigned long long *st) {
        if (!act || b >= 15) return;
        const int off = PK == PK_CP ? p.cp_off : 0;
        if (PK == PK_MRP) {
            tally(st, g + b, (uint32_t)(popc64(K[0]) + popc64(K[1])), (uint32_t)(popc64(Y[0]) + popc64(Y[1])));
        } else {
            stats_ctx(st, off, b);
        }
    }
    BPC_FI void stats_ctx(unsigned long long *st, int off, int b) {
#pragma unroll 1
        for (int k = 0; k < 9; k++) {
            uint32_t n = 0, ones = 0;
#pragma unroll
            for (int c = 0; c < 2; c++) {
                uint64_t m = K[c];
#pragma unroll
                for (int q = 0; q < 4; q++) m &= ((k >> q) & 1) ? cs[c][q] : ~cs[c][q];
                n += (uint32_t)popc64(m);
                ones += (uint32_t)popc64(m & Y[c]);
            }
            tally(st, off + p.a_sig + (g + b) * 9 + k, n, ones);
        }
#pragma unroll 1
        for (int k = 0; k < 4; k++) {
            uint32_t n = 0, ones = 0;
#pragma unroll
            for (int c = 0; c < 2; c++) {
                const uint64_t m = NS[c] & ((k & 1) ? si[c][0] : ~si[c][0]) & ((k & 2) ? si[c][1] : ~si[c][1]);
                n += (uint32_t)popc64(m);
                ones += (uint32_t)popc64(m & sg[c]);
            }
            tally(st, off + p.a_sign + (g + b) * 4 + k, n, ones);
        }
    }
    template <int PK>
    BPC_FI void train_pass(int b, bool act, unsigned long long *st) {
        enc_pass_masks<PK>(b, act);
        stats_pass<PK>(b, act, st);
        enc_pass_commit<PK>(act);
    }

    // ------------------------------------------------------ codeblock driver
    // STATS (encoder only): gather LUT training counts into `stats` instead of
    // writing the slot stream.
    template <bool STATS = false>
    BPC_FI void run(int cb_first, unsigned long long *stats = nullptr) {
        const int grp = lane / G::NL;
        const int cb = cb_first + grp;
        const bool ok = cb < p.cb_end;
        const int cbx = ok ? cb % p.ncbx : 0, cby = ok ? cb / p.ncbx : 0;
        const int x = cbx * CBS + 2 * gl, y0 = cby * CBS;
        g = lut_group(p, x, y0);
        for (int k = 0; k < 2; k++) s.S[k] = s.R[k] = s.N[k] = 0ull;
        s.C[0] = s.C[1] = PASSES == 3 ? G::ROWS : 0ull;  // CP flag at start (:34-39, :73-78)
        s.XL = s.XR = s.XNL = s.XNR = 0ull;
        s.lower = s.size = s.resv = s.cw = 0u;
        s.cnt = 0u;
        s.status = 0;
        s.open_slot = -1;
        s.cur_ev = kEvOpen;
        s.nev = 0;
        XLS = XRS = XLN = XRN = 0ull;
        for (int k = 0; k < 8; k++) evmask[8 * lane + k] = 0u;
        w.sync();
        const size_t cap = (size_t)G::CAP;
        const int32_t *src = p.in + (size_t)y0 * (size_t)p.X + (size_t)x;
        msb = -1;
        top = -1;
        {
            slot_out = p.out + (ok ? (size_t)cb * cap : 0);
            // Read_Coefficients :14-44 + Find_MSB :114-161 in one read: per
            // 32-row half, one 8-byte load per row gives the lane's two
            // columns; signs go to N, magnitudes through a 32x32 bit
            // transpose to bitplanes 0..27 (those up to the quarter's own
            // highest set bit are stored)
            uint32_t mx = 0;
            qtop = 0u;
            if (ok) {
#pragma unroll 1
                for (int h = 0; h < NH; h++) {
                    uint32_t a0[32], a1[32], o0 = 0, o1 = 0, n0 = 0, n1 = 0;
#pragma unroll
                    for (int r = 0; r < 32; r++) {
                        int32_t v0, v1;
                        w.load2(src + (size_t)(h * 32 + r) * (size_t)p.X, v0, v1);
                        a0[r] = v0 < 0 ? 0u - (uint32_t)v0 : (uint32_t)v0;
                        a1[r] = v1 < 0 ? 0u - (uint32_t)v1 : (uint32_t)v1;
                        n0 |= (uint32_t)(v0 < 0) << r;
                        n1 |= (uint32_t)(v1 < 0) << r;
                        o0 |= a0[r];
                        o1 |= a1[r];
                    }
                    s.N[0] |= (uint64_t)n0 << (32 * h);
                    s.N[1] |= (uint64_t)n1 << (32 * h);
                    mx |= o0 | o1;
                    const int t0 = o0 ? 31 - clz32(o0) : -1, t1 = o1 ? 31 - clz32(o1) : -1;
                    qtop |= (uint32_t)(t0 + 1) << (8 * h) | (uint32_t)(t1 + 1) << (8 * (2 + h));
                    transpose32(a0);
#pragma unroll
                    for (int k = 0; k < 28; k++)
                        if (k <= t0) planes[k][h] = a0[k];
                    transpose32(a1);
#pragma unroll
                    for (int k = 0; k < 28; k++)
                        if (k <= t1) planes[k][2 + h] = a1[k];
                }
            }
            if (mx >= (1u << 28)) s.status |= ST_INPUT_RANGE;
            for (int o = G::NL / 2; o; o >>= 1) mx |= w.shfl_xor(mx, o);
            if (ok) {
                msb = mx ? 31 - clz32(mx) : 32;
                if (gl == 0 && !STATS) slot_out[0] = msb;  // :1155
                top = msb <= 27 ? msb : -1;  // planes >= 28 are flag bits, not magnitudes
            }
            // neighbour sign columns are data: lane-1's right, lane+1's left
            const uint64_t up = shfl_up64(w, s.N[1]), dn = shfl_down64(w, s.N[0]);
            s.XNL = gl > 0 ? up : 0ull;
            s.XNR = gl < G::NL - 1 ? dn : 0ull;
        }
        // planes, aligned across the codeblocks that share the warp
        int bmax = msb;
        for (int o = 16; o; o >>= 1) {
            const int other = (int)w.shfl_xor((uint32_t)bmax, o);
            bmax = other > bmax ? other : bmax;
        }
        for (int b = bmax; b >= 0; b--) {
            // 2-pass: planes MSB..0 run SPP, MRP.  3-pass: plane MSB runs CP
            // only, planes below run SPP, MRP, CP (:986-1018).
            const bool full = PASSES == 2 ? b <= msb : b < msb;
            const bool first_cp = PASSES == 3 && b == msb;
            plane_begin(b);
            if (STATS) {
                if (w.any(full)) {
                    train_pass<PK_SPP>(b, full, stats);
                    train_pass<PK_MRP>(b, full, stats);
                }
                if (PASSES == 3 && w.any(full || first_cp)) train_pass<PK_CP>(b, full || first_cp, stats);
            } else {
                if (w.any(full)) {
                    enc_pass<PK_SPP>(b, full);
                    enc_pass<PK_MRP>(b, full);
                }
                if (PASSES == 3 && w.any(full || first_cp)) enc_pass<PK_CP>(b, full || first_cp);
            }
        }
        {
            if (ok && !STATS) {
                if (s.size != 0) {  // flush :1020 (a finished codeword is already stored)
                    if ((uint32_t)s.open_slot < (uint32_t)G::CAP)
                        slot_out[s.open_slot] = (int32_t)s.lower;
                    else
                        s.status |= ST_OVERFLOW;
                }
                // the rest of the slot keeps the -1 fill of :1284
                for (uint32_t k = s.cnt + 1u + (uint32_t)gl; k < (uint32_t)G::CAP; k += G::NL) slot_out[k] = -1;
                if (s.cnt + 1u > (uint32_t)G::CAP) s.status |= ST_OVERFLOW;
            }
        }
        if (ok && p.counts && gl == 0) p.counts[cb] = (int)s.cnt;
        int st = s.status;
        for (int o = 16; o; o >>= 1) st |= (int)w.shfl_xor((uint32_t)st, o);
        if (st && lane == 0 && p.status) w.atomic_or(p.status, st);
    }
};


}  // namespace bpc
