// Tier-1 context modelling of one code-block by one warp (T.800 Annex D; included by t1enc.cu inside
// its anonymous namespace): the (context, decision) symbols of the serial coder, in its order.
//
// An encoder knows every bit beforehand, so all of a pass follows from bitmaps at once, except which
// samples the propagation pass reaches.  Two layouts of the bitmaps are used side by side:
//   rows    a lane holds the four row masks of its stripe (the lanes of a stripe hold the same).
//           The propagation pass's newly significant samples are the least fixpoint of
//             N(c,j) = M(c,j) & (E(c,j) | N(c-1,j-1) | N(c-1,j) | N(c-1,j+1) | N(c,j-1)),
//           found for all stripes together: run fills along the rows by carry propagation, the
//           stripe above's last row taken over by a shuffle, until no lane changes.
//   nibbles a word holds 8 columns x 4 stripe rows, a nibble per column: its bits are in scan
//           order.  A lane holds NW consecutive words, and the lanes hold the block in scan order.
// In the second one the eight neighbours of all 32 samples of a word are eight shifted words (what
// has been scanned already taken with this pass's new samples, the rest without), and the context
// labels come out as four bit slices by logic on whole words; sign contexts likewise.  Each lane
// then writes the symbols of its samples into shared memory at an offset from one prefix sum per
// pass, and the warp copies them out in 16-byte chunks.

template <typename T>
__device__ __forceinline__ T dil(T m) { return m | (T)(m << 1) | (T)(m >> 1); }

// bytes r = 0..3 of x (stripe rows of 8 columns) to nibbles: bit 8r + c to bit 4c + r
__device__ __forceinline__ uint32_t rows_to_nibbles(uint32_t x) {
    uint32_t t;
    t = (x ^ (x >> 12)) & 0x0000F0F0u; x ^= t ^ (t << 12);
    t = (x ^ (x >> 6)) & 0x00CC00CCu; x ^= t ^ (t << 6);
    t = (x ^ (x >> 3)) & 0x0A0A0A0Au; x ^= t ^ (t << 3);
    t = (x ^ (x >> 1)) & 0x22222222u; x ^= t ^ (t << 1);
    return x;
}

__device__ __forceinline__ uint32_t bit_of(uint32_t x, int i) { return (x >> i) & 1u; }

constexpr int kStage = 6144;  // symbols staged per warp and round, after up to 15 left over

struct SymSmem {
    uint4 stage[(kStage + 16) / 16];
    uint32_t neg[4][4][32];  // signs of the left, right, upper, lower neighbours: [which][word][lane]
};

// The eight neighbour words of one word: w, e, n, s and the diagonals
struct Near {
    uint32_t w, e, n, s, nw, ne, sw, se;
    __device__ __forceinline__ uint32_t any() const { return w | e | n | s | nw | ne | sw | se; }
};

// Zero-coding labels (T.800 Table D.1) as four bit slices
__device__ __forceinline__ void zc_slices(const Near& a, int orient, uint32_t (&L)[4]) {
    const uint32_t d1 = a.nw | a.ne | a.sw | a.se;
    const uint32_t t1 = a.nw & a.ne, t0 = a.nw ^ a.ne, b1 = a.sw & a.se, b0 = a.sw ^ a.se;
    const uint32_t d2 = t1 | b1 | (t0 & b0);
    if (orient == J2K_BAND_HH) {
        const uint32_t d3 = (t1 & (a.sw | a.se)) | (b1 & (a.nw | a.ne));
        const uint32_t hv1 = a.w | a.e | a.n | a.s;
        const uint32_t hv2 = (a.w & a.e) | (a.n & a.s) | ((a.w | a.e) & (a.n | a.s));
        const uint32_t two = d2 & ~d3, one = d1 & ~d2;
        L[3] = d3;
        L[2] = two | (one & hv1);
        L[1] = two | (one & ~hv1) | (~d1 & hv2);
        L[0] = (two & hv1) | (one & (hv2 | ~hv1)) | (~d1 & hv1 & ~hv2);
        return;
    }
    const bool hl = orient == J2K_BAND_HL;  // horizontally high-pass: the roles of h and v change
    const uint32_t h_a = hl ? a.n : a.w, h_b = hl ? a.s : a.e, v_a = hl ? a.w : a.n, v_b = hl ? a.e : a.s;
    const uint32_t h2 = h_a & h_b, h1 = h_a ^ h_b, h0 = ~(h_a | h_b);
    const uint32_t v2 = v_a & v_b, v1 = v_a ^ v_b, va = v_a | v_b;
    L[3] = h2;
    L[2] = h1 | (h0 & v2);
    L[1] = (h1 & (va | d1)) | (h0 & (v1 | (~va & d2)));
    L[0] = (h1 & (va | ~d1)) | (h0 & (v1 | (~va & d1 & ~d2)));
}

// Sign-coding symbols (T.800 Tables D.2 and D.3): bits 2..0 of the label (bit 3 is set), the XOR
// bit and the decision, as slices
struct SignSlices {
    uint32_t b2, b1, b0, x, d;
    __device__ __forceinline__ uint32_t symbol(int i) const {
        return 8u | (bit_of(b2, i) << 2) | (bit_of(b1, i) << 1) | bit_of(b0, i) | (bit_of(x, i) << 5) |
               (bit_of(d, i) << 7);
    }
};
__device__ __forceinline__ SignSlices sign_slices(const Near& a, uint32_t own, uint32_t nl, uint32_t nr, uint32_t nu,
                                                  uint32_t nd) {
    const uint32_t wp = a.w & ~nl, wn = a.w & nl, ep = a.e & ~nr, en = a.e & nr;
    const uint32_t np = a.n & ~nu, nn = a.n & nu, sp = a.s & ~nd, sn = a.s & nd;
    const uint32_t hp = (wp & ~en) | (ep & ~wn), hn = (wn & ~ep) | (en & ~wp);
    const uint32_t vp = (np & ~sn) | (sp & ~nn), vn = (nn & ~sp) | (sn & ~np);
    const uint32_t hnz = hp | hn, vnz = vp | vn;
    const uint32_t against = (hn & vp) | (hp & vn);  // the vertical contribution once h is made positive
    SignSlices r;
    r.b2 = hnz & ~against;
    r.b1 = against | (~hnz & vnz);
    r.b0 = ~(hnz ^ vnz);
    r.x = hn | (~hnz & vn);
    r.d = own ^ r.x;
    return r;
}

// NW words per lane, LPS lanes per stripe, RT row masks of 8 * NW * LPS columns or more.
// NARROW: a stripe is one word, which all its lanes hold; each writes the symbols of 32 / LPS samples.
// Such blocks are small: what counts is not their symbols but what every plane and pass costs whatever
// it holds, so the empty passes and exchanges are left out (at most 8 x 64 samples, whose symbols of a
// pass fit the stage).
template <int NW, int LPS, typename RT, bool NARROW = false>
__device__ __forceinline__ void symbols_of_block(SymSmem& S, const j2k_cb_job& J, int jid, int lane,
                                                 const int32_t* __restrict__ coeff, uint8_t* __restrict__ syms,
                                                 uint32_t* __restrict__ nsyms, uint32_t* __restrict__ pass_end,
                                                 uint64_t* __restrict__ planes, j2k_cb_desc* __restrict__ descs,
                                                 uint32_t* __restrict__ err, int pad) {
    constexpr unsigned FULL = 0xffffffffu;
    static_assert(!NARROW || NW == 1, "");
    constexpr bool kOne = LPS == 32;  // one stripe
    const int cw = J.cw, ch = J.ch, orient = J.orient;
    const int32_t* blk = coeff + J.off;
    constexpr int SEG = 32 / LPS;  // the lane's samples of a narrow word, and those before them
    const uint32_t before_me = (1u << (SEG * (lane % LPS))) - 1u;
    const uint32_t me = (SEG == 32 ? ~0u : (1u << (SEG & 31)) - 1u) << (SEG * (lane % LPS));
    const int s0 = 4 * (lane / LPS), part = NARROW ? 0 : lane % LPS;  // first row of the lane's stripe, place in it

    // ---- bit-plane slicing: lane p ends up holding plane p of each row and stores it (one word: lane i
    // holds sample i, and a plane is one vote)
    uint32_t mor = 0, mine_abs = 0;
    bool mine_neg = false;
    const bool mine_in = (lane & 3) < ch && lane >> 2 < cw;
    if constexpr (kOne) {
        const int32_t v = mine_in ? blk[(size_t)(lane & 3) * J.pitch + (lane >> 2)] : 0;
        mine_neg = v < 0;
        mor = mine_abs = v < 0 ? (uint32_t)(-(int64_t)v) : (uint32_t)v;
    }
    constexpr int G = 4;  // rows whose loads are in flight together
    for (int r0 = 0; r0 < ch && !kOne; r0 += G) {
        int32_t a0[G], a1[G];
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const int32_t* row = blk + (size_t)(r0 + g) * J.pitch;
            a0[g] = r0 + g < ch && lane < cw ? row[lane] : 0;
            a1[g] = sizeof(RT) == 8 && r0 + g < ch && lane + 32 < cw ? row[lane + 32] : 0;
        }
#pragma unroll
        for (int g = 0; g < G; ++g) {
            if (r0 + g >= ch) break;
            const uint32_t m0 = a0[g] < 0 ? (uint32_t)(-(int64_t)a0[g]) : (uint32_t)a0[g];
            const uint32_t m1 = a1[g] < 0 ? (uint32_t)(-(int64_t)a1[g]) : (uint32_t)a1[g];
            RT ng = (RT)__ballot_sync(FULL, a0[g] < 0);
            if (sizeof(RT) == 8) ng |= (RT)((uint64_t)__ballot_sync(FULL, a1[g] < 0) << 32);
            mor |= m0 | m1;
            const uint32_t any = __reduce_or_sync(FULL, m0 | m1);
            uint64_t mine = 0;
            for (int p = 0; p < 32 && (any >> p); ++p) {
                uint64_t pm = __ballot_sync(FULL, (m0 >> p) & 1);
                if (sizeof(RT) == 8) pm |= (uint64_t)__ballot_sync(FULL, (m1 >> p) & 1) << 32;
                if (lane == p) mine = pm;
            }
            if (lane == 31) mine = ng;  // signs in the place of plane 31, which no block has (see below)
            planes[(r0 + g) * 32 + lane] = mine;  // [row][plane]: one coalesced 256-byte store
        }
    }
    mor = __reduce_or_sync(FULL, mor);
    const int numbps = mor ? 32 - __clz(mor) : 0;
    j2k_cb_desc d;
    d.offset = (uint32_t)J.out_off;
    d.length = 0;
    d.numbps = (uint8_t)numbps;
    d.npasses = (uint8_t)(numbps ? 3 * numbps - 2 : 0);
    d.orient = J.orient;
    d.band = J.band;
    d.x0 = J.px0;
    d.y0 = J.py0;
    d.cw = J.cw;
    d.ch = J.ch;
    d.comp = J.comp;
    d.reserved = 0;
    if (numbps > 31) {
        if (lane == 0) {
            atomicCAS(err, 0u, (uint32_t)J2K_DEVERR_PLANES);
            nsyms[jid] = 0;
            descs[jid] = d;
        }
        __syncwarp();
        return;
    }
    __syncwarp();

    // a word from the lane of the stripe above / below or of the words before / after (0 outside)
    auto above = [&](uint32_t x) {
        if constexpr (kOne) return 0u;
        const uint32_t t = __shfl_up_sync(FULL, x, LPS);
        return lane < LPS ? 0u : t;
    };
    auto below = [&](uint32_t x) {
        if constexpr (kOne) return 0u;
        const uint32_t t = __shfl_down_sync(FULL, x, LPS);
        return lane >= 32 - LPS ? 0u : t;
    };
    auto before = [&](uint32_t x) {
        if constexpr (NARROW) return 0u;
        const uint32_t t = __shfl_up_sync(FULL, x, 1);
        return part == 0 ? 0u : t;
    };
    auto after = [&](uint32_t x) {
        if constexpr (NARROW) return 0u;
        const uint32_t t = __shfl_down_sync(FULL, x, 1);
        return part == LPS - 1 ? 0u : t;
    };
    // the lane's words of four row masks
    auto nibbles = [&](const RT (&row)[4], uint32_t (&x)[NW]) {
        uint32_t h[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) h[j] = (uint32_t)(row[j] >> (part * NW * 8));
#pragma unroll
        for (int k = 0; k < NW; ++k) {
            const uint32_t lo = __byte_perm(h[0], h[1], k | ((4 + k) << 4));  // byte k of rows 0 and 1
            const uint32_t hi = __byte_perm(h[2], h[3], k | ((4 + k) << 4));
            x[k] = rows_to_nibbles(__byte_perm(lo, hi, 0x5410));
        }
    };

    // the samples of the block that the lane's words hold, and its rows
    uint32_t V[NW], sig[NW], ref[NW], neg[NW];
    RT Vr[4], O[4], negrow[4];
    const RT colmask = cw >= (int)sizeof(RT) * 8 ? (RT) ~(RT)0 : (RT)(((RT)1 << cw) - 1);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        Vr[j] = s0 + j < ch ? colmask : (RT)0;
        O[j] = 0;
        negrow[j] = !kOne && s0 + j < ch ? (RT)planes[(s0 + j) * 32 + 31] : (RT)0;
    }
    if constexpr (kOne) {
        V[0] = __ballot_sync(FULL, mine_in);
        neg[0] = __ballot_sync(FULL, mine_neg);
    } else {
        nibbles(Vr, V);
        nibbles(negrow, neg);
    }
    {  // signs of the four direct neighbours
        const uint32_t pv = before(neg[NW - 1]), nx = after(neg[0]);
#pragma unroll
        for (int k = 0; k < NW; ++k) {
            S.neg[0][k][lane] = (neg[k] << 4) | ((k ? neg[k ? k - 1 : 0] : pv) >> 28);
            S.neg[1][k][lane] = (neg[k] >> 4) | ((k < NW - 1 ? neg[k < NW - 1 ? k + 1 : k] : nx) << 28);
            S.neg[2][k][lane] = ((neg[k] << 1) & 0xEEEEEEEEu) | ((above(neg[k]) >> 3) & 0x11111111u);
            S.neg[3][k][lane] = ((neg[k] >> 1) & 0x77777777u) | ((below(neg[k]) << 3) & 0x88888888u);
            sig[k] = 0;
            ref[k] = 0;
        }
    }

    // Neighbour words of all the lane's words: xo the significance before this pass, xn after it.
    // Scanned before a sample: the stripe above, its own column's rows above, the column to the left.
    auto neighbours = [&](const uint32_t (&xo)[NW], const uint32_t (&xn)[NW], Near (&a)[NW]) {
        uint32_t un[NW], dn[NW], uo[NW], dol[NW];
#pragma unroll
        for (int k = 0; k < NW; ++k) {
            const uint32_t top = (above(xn[k]) >> 3) & 0x11111111u, bot = (below(xo[k]) << 3) & 0x88888888u;
            un[k] = ((xn[k] << 1) & 0xEEEEEEEEu) | top;
            uo[k] = ((xo[k] << 1) & 0xEEEEEEEEu) | top;
            dn[k] = ((xn[k] >> 1) & 0x77777777u) | bot;
            dol[k] = ((xo[k] >> 1) & 0x77777777u) | bot;
        }
        const uint32_t pu = before(un[NW - 1]), px = before(xn[NW - 1]), pd = before(dn[NW - 1]);
        const uint32_t nu = after(uo[0]), nx = after(xo[0]), nd = after(dol[0]);
#pragma unroll
        for (int k = 0; k < NW; ++k) {
            a[k].nw = __funnelshift_l(k ? un[k ? k - 1 : 0] : pu, un[k], 4);
            a[k].w = __funnelshift_l(k ? xn[k ? k - 1 : 0] : px, xn[k], 4);
            a[k].sw = __funnelshift_l(k ? dn[k ? k - 1 : 0] : pd, dn[k], 4);
            a[k].n = un[k];
            a[k].s = dol[k];
            a[k].ne = __funnelshift_r(uo[k], k < NW - 1 ? uo[k < NW - 1 ? k + 1 : k] : nu, 4);
            a[k].e = __funnelshift_r(xo[k], k < NW - 1 ? xo[k < NW - 1 ? k + 1 : k] : nx, 4);
            a[k].se = __funnelshift_r(dol[k], k < NW - 1 ? dol[k < NW - 1 ? k + 1 : k] : nd, 4);
        }
    };
    auto signs = [&](const Near& a, int k) {
        return sign_slices(a, neg[k], S.neg[0][k][lane], S.neg[1][k][lane], S.neg[2][k][lane], S.neg[3][k][lane]);
    };

    uint8_t* out = syms + J.sym_off;
    uint32_t* pend = pass_end + (size_t)jid * 92;
    uint8_t* stage = reinterpret_cast<uint8_t*>(S.stage);
    const int cap = (int)J.sym_cap;
    int pos = 0, npass = 0;
    bool ovf = false;
    // One pass's symbols: each lane has cnt of them, which emit(at) writes from stage[at] on.  The
    // stage holds the bytes from the last 16-byte boundary of the output on.
    auto write_pass = [&](int cnt, auto emit) {
        int tot = cnt, off = 0;
        if (NARROW && !kOne) {  // every lane of a stripe has its count
            off = warp_excl(lane % LPS == 0 ? cnt : 0, lane, &tot);
            if (lane % LPS != 0) off -= cnt;
        } else if (!kOne) {
            off = warp_excl(cnt, lane, &tot);
        }
        if (pos + tot > cap) {
            ovf = true;
            return;
        }
        for (int base = 0; base < tot;) {  // lanes whose symbols fit the stage (at most 320 a lane)
            const bool mine = off >= base && off + cnt <= base + kStage && cnt > 0;
            const int lead = pos & 15;
            if (mine) emit(lead + off - base);
            const unsigned left = NARROW ? 0u : __ballot_sync(FULL, cnt > 0 && off + cnt > base + kStage);
            const int next = left ? __shfl_sync(FULL, off, __ffs(left) - 1) : tot;
            __syncwarp();
            const int fill = lead + next - base, full = fill >> 4;
            if (!NARROW || full > 0) {
                uint4* dst = reinterpret_cast<uint4*>(out + (pos - lead));
                for (int i = lane; i < full; i += 32) dst[i] = S.stage[i];
                const uint4 rest = S.stage[full];
                __syncwarp();
                if (lane == 0) S.stage[0] = rest;
                __syncwarp();
            }
            pos += next - base;
            base = next;
        }
    };
    // writes the bytes after the last 16-byte boundary out too (a whole chunk: capacities are
    // multiples of 16); the stage still holds them
    auto write_rest = [&]() {
        if ((pos & 15) && lane == 0) reinterpret_cast<uint4*>(out)[pos >> 4] = S.stage[0];
    };
    auto end_pass = [&]() {
        if (lane == 0) pend[npass] = (uint32_t)pos;
        ++npass;
        if (pad) {  // the next pass starts on a 16-byte boundary (a coding unit of its own)
            if (!ovf) write_rest();
            __syncwarp();  // before another lane writes the stage's first bytes again
            pos = (pos + 15) & ~15;
            ovf |= pos > cap;
        }
    };

    bool all = false;  // every sample is significant: the propagation and cleanup passes are empty
    for (int p = numbps - 1; p >= 0 && !ovf; --p) {
        RT Br[4];
        uint32_t B[NW], K[NW], now[NW];  // this plane, samples the propagation pass codes, significance
#pragma unroll
        for (int j = 0; j < 4; ++j) Br[j] = !kOne && s0 + j < ch ? (RT)planes[(s0 + j) * 32 + p] : (RT)0;
        if constexpr (kOne) B[0] = __ballot_sync(FULL, (mine_abs >> p) & 1u);
        else nibbles(Br, B);
#pragma unroll
        for (int k = 0; k < NW; ++k) {
            K[k] = 0;
            now[k] = sig[k];
        }
        if (p != numbps - 1) {
            // ------------------------- significance propagation pass
            Near a[NW];
            int cnt = 0;
            if (!all) {
                uint32_t Nn[NW];
                if constexpr (NARROW) {  // on the words themselves, a step a sample: they are short
                    neighbours(sig, sig, a);
                    const uint32_t M = V[0] & ~sig[0] & B[0];
                    uint32_t N = M & a[0].any(), was;
                    do {
                        was = N;
                        const uint32_t top = (above(N) >> 3) & 0x11111111u, un = ((N << 1) & 0xEEEEEEEEu) | top;
                        N |= M & (un | (un << 4) | (top >> 4) | (N << 4) | ((N << 3) & 0x77777777u));
                    } while (kOne ? N != was : __any_sync(FULL, N != was));
                    Nn[0] = N;
                } else {
                    RT N[4] = {0, 0, 0, 0};
                    RT up = __shfl_up_sync(FULL, O[3], LPS), dw = __shfl_down_sync(FULL, O[0], LPS);
                    if (lane < LPS) up = 0;
                    if (lane >= 32 - LPS) dw = 0;
                    RT E[4], M[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const RT u = j ? O[j ? j - 1 : 0] : up, w = j < 3 ? O[j < 3 ? j + 1 : 3] : dw;
                        M[j] = Vr[j] & ~O[j] & Br[j];
                        E[j] = M[j] & dil((RT)(u | O[j] | w));
                    }
                    bool more;
                    do {
                        RT ab = __shfl_up_sync(FULL, N[3], LPS);
                        if (lane < LPS) ab = 0;
                        RT was = 0;
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const RT u = j ? N[j ? j - 1 : 0] : (RT)0, w = j < 3 ? N[j < 3 ? j + 1 : 3] : (RT)0;
                            const RT seeds = (E[j] | (M[j] & ((RT)((u | w) << 1) | u | (j == 0 ? dil(ab) : (RT)0))));
                            const RT f = M[j] & ((RT) ~(RT)(M[j] + seeds) | seeds);
                            was |= f ^ N[j];
                            N[j] = f;
                        }
                        more = __any_sync(FULL, was != 0);
                    } while (more);
                    nibbles(N, Nn);
                }
#pragma unroll
                for (int k = 0; k < NW; ++k) now[k] = sig[k] | Nn[k];
                neighbours(sig, now, a);
#pragma unroll
                for (int k = 0; k < NW; ++k) {
                    K[k] = V[k] & ~sig[k] & a[k].any();
                    cnt += __popc(K[k]) + __popc(Nn[k]);
                }
                write_pass(cnt, [&](int at) {
#pragma unroll
                    for (int k = 0; k < NW; ++k) {
                        uint32_t L[4], m = K[k];
                        if (!m) continue;
                        if (NARROW) at += __popc(m & before_me) + __popc(m & B[k] & before_me), m &= me;
                        zc_slices(a[k], orient, L);
                        const SignSlices g = signs(a[k], k);
                        while (m) {
                            const int i = __ffs((int)m) - 1;
                            m &= m - 1;
                            const uint32_t b = bit_of(B[k], i);
                            stage[at++] = (uint8_t)(bit_of(L[0], i) | (bit_of(L[1], i) << 1) | (bit_of(L[2], i) << 2) |
                                                    (bit_of(L[3], i) << 3) | (b << 7));
                            if (b) stage[at++] = (uint8_t)g.symbol(i);
                        }
                    }
                });
            }
            end_pass();
            if (ovf) break;
            // ------------------------- magnitude refinement pass
            neighbours(now, now, a);
            cnt = 0;
#pragma unroll
            for (int k = 0; k < NW; ++k) cnt += __popc(sig[k]);
            write_pass(cnt, [&](int at) {
#pragma unroll
                for (int k = 0; k < NW; ++k) {
                    const uint32_t nb = a[k].any();
                    uint32_t m = sig[k];
                    if (NARROW) at += __popc(m & before_me), m &= me;
                    while (m) {
                        const int i = __ffs((int)m) - 1;
                        m &= m - 1;
                        stage[at++] = (uint8_t)((bit_of(ref[k], i) ? 16u : 14u | bit_of(nb, i)) | (bit_of(B[k], i) << 7));
                    }
                }
            });
#pragma unroll
            for (int k = 0; k < NW; ++k) ref[k] = sig[k];
            end_pass();
            if (ovf) break;
        }
        // ------------------------- cleanup pass
        if (!all) {
            uint32_t C[NW], fin[NW];
            Near a[NW];
#pragma unroll
            for (int k = 0; k < NW; ++k) {
                C[k] = V[k] & ~now[k] & ~K[k];
                fin[k] = now[k] | (C[k] & B[k]);
            }
            neighbours(now, fin, a);
            int cnt = 0;
            uint32_t ev[NW], run[NW];  // samples with a symbol; those that start a run-length column
#pragma unroll
            for (int k = 0; k < NW; ++k) {
                // run-length columns: four samples to code and, before the column, no significant one
                // around it (its own rows are insignificant then; the rows above and below it count)
                const uint32_t side = a[k].w | a[k].e | a[k].nw | a[k].ne | a[k].sw | a[k].se |
                                      (a[k].n & 0x11111111u) | (a[k].s & 0x88888888u);
                uint32_t q = C[k] & ~side;
                q &= (q >> 1);
                q &= (q >> 2) & 0x11111111u;
                const uint32_t col = q * 15u, x = B[k] & col;
                const uint32_t some = (x | (x >> 1) | (x >> 2) | (x >> 3)) & q;  // columns with a 1
                const uint32_t fst = x & ~(((x << 1) & 0xEEEEEEEEu) | ((x << 2) & 0xCCCCCCCCu) | ((x << 3) & 0x88888888u));
                run[k] = fst | (q & ~some);
                ev[k] = (C[k] & ~col) | run[k] | (fst << 1 & 0xEEEEEEEEu) | (fst << 2 & 0xCCCCCCCCu) |
                        (fst << 3 & 0x88888888u);
                cnt += __popc(ev[k]) + __popc(ev[k] & B[k]) + 2 * __popc(fst);
            }
            write_pass(cnt, [&](int at) {
#pragma unroll
                for (int k = 0; k < NW; ++k) {
                    uint32_t L[4], m = ev[k];
                    if (!m) continue;
                    if (NARROW)
                        at += __popc(m & before_me) + __popc(m & B[k] & before_me) + 2 * __popc(run[k] & B[k] & before_me),
                            m &= me;
                    zc_slices(a[k], orient, L);
                    const SignSlices g = signs(a[k], k);
                    while (m) {
                        const int i = __ffs((int)m) - 1;
                        m &= m - 1;
                        const uint32_t b = bit_of(B[k], i);
                        uint32_t v = bit_of(L[0], i) | (bit_of(L[1], i) << 1) | (bit_of(L[2], i) << 2) | (bit_of(L[3], i) << 3);
                        const uint32_t r = bit_of(run[k], i);
                        if (r) v = 17u;
                        stage[at++] = (uint8_t)(v | (b << 7));
                        if (r & b) {  // the row of the first 1, two bits
                            stage[at++] = (uint8_t)(18u | ((uint32_t)(i & 2) << 6));
                            stage[at++] = (uint8_t)(18u | ((uint32_t)(i & 1) << 7));
                        }
                        if (b) stage[at++] = (uint8_t)g.symbol(i);
                    }
                }
            });
            uint32_t none = 0;
#pragma unroll
            for (int k = 0; k < NW; ++k) {
                sig[k] = fin[k];
                none |= V[k] & ~sig[k];
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) O[j] |= Br[j] & Vr[j];
            if (NARROW) all = !__any_sync(FULL, none != 0);
        }
        end_pass();
    }
    if (ovf) {
        if (lane == 0) atomicCAS(err, 0u, (uint32_t)J2K_DEVERR_SYM_CAPACITY);
        pos = 0;
    } else if (!pad) {
        write_rest();
    }
    if (lane == 0) {
        nsyms[jid] = (uint32_t)pos;
        descs[jid] = d;
    }
    __syncwarp();
}

#define SYMBOLS_ARGS                                                                                                    \
    SymSmem &S, const j2k_cb_job &J, int jid, int lane, const int32_t *__restrict__ coeff, uint8_t *__restrict__ syms, \
        uint32_t *__restrict__ nsyms, uint32_t *__restrict__ pass_end, uint64_t *__restrict__ planes,                  \
        j2k_cb_desc *__restrict__ descs, uint32_t *__restrict__ err, int pad
#define SYMBOLS(...) __VA_ARGS__(S, J, jid, lane, coeff, syms, nsyms, pass_end, planes, descs, err, pad)

// a call of its own, so that the common forms' code is what it would be without this one
template <int NW, int LPS, typename RT, bool NARROW = false>
__device__ __noinline__ void symbols_of_rare_block(SYMBOLS_ARGS) {
    SYMBOLS(symbols_of_block<NW, LPS, RT, NARROW>);
}

// The form that keeps most lanes busy: 32 / LPS stripes of 8 * NW * LPS columns, or for narrow blocks of
// one word each.  Bound by issue.  Whole encodes of 2048 x 2048 colour with three forms only (wider than
// 32, narrower, at most 32 x 32) -> with these: blocks of 64 x 4 2.80 -> 1.24 ms, 64 x 8 1.84 -> 0.98, 8 x 8
// 2.92 -> 1.77, 4 x 4 6.62 -> 2.88; 32 x 32 and 64 x 64 as before.
__device__ __forceinline__ void symbols_of_shape(SYMBOLS_ARGS) {
    const int w = J.cw, h = J.ch;
    if (w <= 8 && h <= 4) SYMBOLS(symbols_of_rare_block<1, 32, uint32_t, true>);
    else if (w <= 8 && h <= 8) SYMBOLS(symbols_of_rare_block<1, 16, uint32_t, true>);
    else if (w <= 8 && h <= 16) SYMBOLS(symbols_of_rare_block<1, 8, uint32_t, true>);
    else if (w <= 8 && h <= 32) SYMBOLS(symbols_of_rare_block<1, 4, uint32_t, true>);
    else if (w <= 8) SYMBOLS(symbols_of_rare_block<1, 2, uint32_t, true>);
    else if (w <= 32 && h <= 32) SYMBOLS(symbols_of_block<1, 4, uint32_t>);
    else if (w <= 32) SYMBOLS(symbols_of_block<2, 2, uint32_t>);
    else if (h <= 16) SYMBOLS(symbols_of_rare_block<1, 8, uint64_t>);
    else if (h <= 32) SYMBOLS(symbols_of_rare_block<2, 4, uint64_t>);
    else SYMBOLS(symbols_of_block<4, 2, uint64_t>);
}
#undef SYMBOLS
#undef SYMBOLS_ARGS
