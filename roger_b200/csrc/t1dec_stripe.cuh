// Tier-1 block decoder, stripe by stripe (T.800 Annex D; included by t1dec.cu inside its anonymous
// namespace, after DecTables).
//
// A warp decodes L code-blocks side by side, lane b the symbols of block b.  The symbols of a block
// form one serial chain, so everything that does not belong to that chain is taken out of it and
// done by the whole warp together, once per pass and stripe of four rows:
//   prepare  turns the block's bitmaps into one 32-bit word per stripe column that holds all the
//            column's symbols need (the 3 x 6 significance neighbourhood and the signs around it, or
//            the refinement labels), and the set of columns that have a symbol;
//   decode   lane b walks its columns in one flat loop, a significance / refinement decision per
//            turn: fetch the next column when the last one is done, decode, update the word in
//            registers (a sample that turns significant reaches the next column as a carry);
//   finish   turns the column words back into the bitmaps.
// The lanes of a warp go through the bit-planes, passes and stripes together, so that they meet on
// the same instructions.  A stripe of a block is Q words of 8 columns: 8, or 1 for blocks that are no
// wider.  Those in the form for 64 columns left seven eighths of the lanes idle while a stripe was
// prepared and finished: host to host on B200, 4096 x 4096 colour with blocks of 4 x 64 42.7 -> 15.4 ms,
// 8 x 8 38.7 -> 16.5, 2048 x 2048 with 4 x 64 12.0 -> 6.3, 1024 x 1024 with 8 x 64 3.6 -> 3.2.
//
// Bitmaps: one word per 8 columns of a stripe, a nibble per column (bit j = stripe row j).
// Column word of the propagation and cleanup passes:
//   bits 0-17   significance, row r = 0..5 (the row above the stripe, its four rows, the row below)
//               at 3r: column x-1, x, x+1
//   bits 18-21  signs of column x-1, stripe rows 0..3
//   bits 22-27  signs of column x, rows above..below
//   bits 28-31  signs of column x+1, stripe rows 0..3
// (a sign bit counts only where the sample is significant).  Column word of the refinement pass:
// per stripe row k at 3k: to refine, refined before, has a significant neighbour.
//
// The parts are host-callable (one lane at a time), which is how they are tested without a GPU.

#define T1D_HD __host__ __device__ __forceinline__

T1D_HD int ctz32(uint32_t v) {  // -1 for 0
#ifdef __CUDA_ARCH__
    return __ffs((int)v) - 1;
#else
    return v ? __builtin_ctz(v) : -1;
#endif
}

T1D_HD int popc32(uint32_t v) {
#ifdef __CUDA_ARCH__
    return __popc(v);
#else
    return __builtin_popcount(v);
#endif
}

// 4 bits to bits 0, 3, 6, 9 and back
T1D_HD uint32_t spread4(uint32_t n) {
    n = (n | (n << 4)) & 0xC3u;
    return (n | (n << 2)) & 0x249u;
}
T1D_HD uint32_t gather4(uint32_t x) {
    x &= 0x249u;
    x = (x | (x >> 2)) & 0xC3u;
    return (x | (x >> 4)) & 0xFu;
}

// MQ state of a context: x = Qe as a float, the MPS in the sign bit; y = Qe << 16 | table entry after
// an LPS << 8 | entry after an MPS (entries of the 94-entry table, state * 2 + MPS)
struct alignas(8) MqdState {
    uint32_t x, y;
};

// Words of a warp's L blocks, interleaved by block so that the lanes' accesses fall in distinct
// banks: four bitmaps of 16 stripes x Q words (blocks of up to 8 * Q columns), 8 * Q column words, 19
// context states of 2 words, 2 words of column sets.
template <int L, int Q>
struct StripeState {
    static constexpr int kMap = 16 * Q, kCols = 4 * kMap, kCtx = kCols + 8 * Q, kSets = kCtx + 38, kWords = kSets + 2;
    uint32_t* w;
    T1D_HD uint32_t& sig(int s, int q, int b) const { return w[(s * Q + q) * L + b]; }
    T1D_HD uint32_t& neg(int s, int q, int b) const { return w[(kMap + s * Q + q) * L + b]; }
    T1D_HD uint32_t& vis(int s, int q, int b) const { return w[(2 * kMap + s * Q + q) * L + b]; }
    T1D_HD uint32_t& ref(int s, int q, int b) const { return w[(3 * kMap + s * Q + q) * L + b]; }
    T1D_HD uint32_t& col(int x, int b) const { return w[(kCols + x) * L + b]; }
    T1D_HD MqdState& ctx(int k, int b) const { return reinterpret_cast<MqdState*>(w + kCtx * L)[k * L + b]; }
    // column set of block b, a byte per 8 columns (the bytes of one block are contiguous)
    T1D_HD uint8_t* cols(int b) const { return reinterpret_cast<uint8_t*>(w + kSets * L) + 8 * b; }
    T1D_HD uint32_t& colset(int h, int b) const { return (w + kSets * L)[2 * b + h]; }
};
template <int L, int Q>
__host__ __device__ constexpr int stripe_state_words() {
    return StripeState<L, Q>::kWords * L;
}

enum : int { kPassSP = 0, kPassMR = 1, kPassCU = 2 };

// rows of a column word (propagation / cleanup) with any significant sample in the 3 x 3 window,
// the centre included, at 3k
T1D_HD uint32_t near_rows(uint32_t W) {
    const uint32_t t = W | (W >> 1) | (W >> 2);
    return t | (t >> 3) | (t >> 6);
}

// prepare: word q (8 columns) of stripe s of block b, whose rows below the block are outside rv (the
// stripe's valid rows at 3k) and whose width is cw
template <int L, int Q>
T1D_HD void stripe_prepare_zc(const StripeState<L, Q>& S, int kind, int s, int q, int b, int cw, uint32_t rv) {
    if (8 * q >= cw) {
        S.cols(b)[q] = 0;
        return;
    }
    uint32_t sg[3][3], ng[3][3];  // [stripe s-1, s, s+1][word q-1, q, q+1]
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const bool in = s + i >= 1 && s + i <= 16 && (Q > 1 ? q + j >= 1 && q + j <= Q : j == 1);
            sg[i][j] = in ? S.sig(s + i - 1, q + j - 1, b) : 0u;
            ng[i][j] = in ? S.neg(s + i - 1, q + j - 1, b) : 0u;
        }
    uint32_t own_ng = ng[1][1];
    if (kind == kPassCU) own_ng |= S.vis(s, q, b) & ~sg[1][1];  // visited samples, see stripe_decode
    // column i - 1 of the word for i = 0 (the word to the left) .. 9 (to the right)
    auto sig_col = [&](int i) -> uint32_t {
        const int j = i == 0 ? 0 : (i == 9 ? 2 : 1), sh = 4 * ((i + 7) & 7);
        return (spread4((sg[1][j] >> sh) & 15u) << 3) | ((sg[0][j] >> (sh + 3)) & 1u) |
               (((sg[2][j] >> sh) & 1u) << 15);
    };
    auto neg_col = [&](int i) -> uint32_t {
        const int j = i == 0 ? 0 : (i == 9 ? 2 : 1), sh = 4 * ((i + 7) & 7);
        return (ng[1][j] >> sh) & 15u;
    };
    uint32_t v0 = sig_col(0), v1 = sig_col(1), n0 = neg_col(0), n1 = neg_col(1), set = 0;
#pragma unroll
    for (int i = 1; i <= 8; ++i) {
        if (Q == 1 && i > cw) break;
        const uint32_t v2 = sig_col(i + 1), n2 = neg_col(i + 1);
        const int sh = 4 * (i - 1);
        const uint32_t vert = ((ng[0][1] >> (sh + 3)) & 1u) | (((own_ng >> sh) & 15u) << 1) |
                              (((ng[2][1] >> sh) & 1u) << 5);
        const uint32_t W = v0 | (v1 << 1) | (v2 << 2) | (n0 << 18) | (vert << 22) | (n2 << 28);
        S.col(8 * q + i - 1, b) = W;
        uint32_t c = ~(W >> 4) & rv;
        if (kind == kPassSP) c &= near_rows(W);
        else c &= ~spread4((W >> 23) & 15u);
        set |= (uint32_t)(c != 0) << (i - 1);
        v0 = v1;
        v1 = v2;
        n0 = n1;
        n1 = n2;
    }
    if (cw - 8 * q < 8) set &= (1u << (cw - 8 * q)) - 1u;
    S.cols(b)[q] = (uint8_t)set;
    if (Q == 1 && kind == kPassSP) S.vis(s, q, b) = 0;  // a stripe without symbols is not finished
}

// The same for one column of a stripe of one word, so that a block's columns can be prepared by as many
// lanes; returns whether the column has a symbol (the caller puts the set together).
template <int L>
T1D_HD bool stripe_prepare_column(const StripeState<L, 1>& S, int kind, int s, int x, int b, uint32_t rv) {
    const uint32_t sg = S.sig(s, 0, b), ng = S.neg(s, 0, b);
    const uint32_t sa = s > 0 ? S.sig(s - 1, 0, b) : 0u, na = s > 0 ? S.neg(s - 1, 0, b) : 0u;
    const uint32_t se = s < 15 ? S.sig(s + 1, 0, b) : 0u, ne = s < 15 ? S.neg(s + 1, 0, b) : 0u;
    uint32_t own_ng = ng;
    if (kind == kPassCU) own_ng |= S.vis(s, 0, b) & ~sg;
    // columns x - 1, x, x + 1 of a word at bits 0, 4, 8
    const auto three = [&](uint32_t w) { return x ? (w >> (4 * x - 4)) & 0xFFFu : (w << 4) & 0xFFFu; };
    const uint32_t m = three(sg), a = three(sa), e = three(se), n = three(ng);
    uint32_t W = 0;
#pragma unroll
    for (int i = 0; i < 3; ++i)
        W |= ((spread4((m >> (4 * i)) & 15u) << 3) | ((a >> (4 * i + 3)) & 1u) | (((e >> (4 * i)) & 1u) << 15)) << i;
    const int sh = 4 * x;
    const uint32_t vert = ((na >> (sh + 3)) & 1u) | (((own_ng >> sh) & 15u) << 1) | (((ne >> sh) & 1u) << 5);
    W |= ((n & 15u) << 18) | (vert << 22) | ((n >> 8) << 28);
    S.col(x, b) = W;
    const uint32_t c = ~(W >> 4) & rv;
    return (kind == kPassSP ? c & near_rows(W) : c & ~spread4((W >> 23) & 15u)) != 0;
}

// samples of word q that the refinement pass codes (significant before this plane), and the number
// of those in the words before it: within a word the bits are in coding order already
template <int L, int Q>
T1D_HD uint32_t stripe_mr_symbols(const StripeState<L, Q>& S, int s, int q, int b, int* before) {
    int n = 0;
    for (int i = 0; i < q; ++i) n += popc32(S.sig(s, i, b) & ~S.vis(s, i, b));
    *before = n;
    return S.sig(s, q, b) & ~S.vis(s, q, b);
}

// prepare of a refinement stripe: no decision changes another one's context here, so the stripe's
// labels are listed in coding order (a byte each, in the column words) and their number put in
// column set word 0
template <int L, int Q>
T1D_HD void stripe_prepare_mr(const StripeState<L, Q>& S, int s, int q, int b, int cw) {
    if (8 * q >= cw) return;
    uint32_t vert = 0, h3[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        const bool in = Q > 1 ? q + j >= 1 && q + j <= Q : j == 1;
        const uint32_t m = in ? S.sig(s, q + j - 1, b) : 0u;
        const uint32_t a = in && s > 0 ? S.sig(s - 1, q + j - 1, b) : 0u;
        const uint32_t e = in && s < 15 ? S.sig(s + 1, q + j - 1, b) : 0u;
        const uint32_t ud = ((m << 1) & 0xEEEEEEEEu) | ((a >> 3) & 0x11111111u) | ((m >> 1) & 0x77777777u) |
                            ((e << 3) & 0x88888888u);
        h3[j] = m | ud;
        if (j == 1) vert = ud;
    }
    const uint32_t nb = vert | (h3[1] << 4) | (h3[0] >> 28) | (h3[1] >> 4) | (h3[2] << 28);
    const uint32_t r = S.ref(s, q, b);
    int at = 0;
    uint32_t m = stripe_mr_symbols(S, s, q, b, &at);
    S.ref(s, q, b) = r | m;
    if (8 * (q + 1) >= cw) S.colset(0, b) = (uint32_t)(at + popc32(m));
    while (m) {
        const int i = ctz32(m);
        m &= m - 1;
        reinterpret_cast<uint8_t*>(&S.col(at >> 2, b))[at & 3] =
            (uint8_t)(((r >> i) & 1u) ? 16u : 14u + ((nb >> i) & 1u));
        ++at;
    }
}

// finish: the decisions of a refinement stripe (32 to a word, in coding order) back to their samples
template <int L, int Q>
T1D_HD uint32_t stripe_finish_mr(const StripeState<L, Q>& S, int s, int q, int b, int cw) {
    if (8 * q >= cw) return 0;
    int at = 0;
    uint32_t ones = 0;
    for (uint32_t m = stripe_mr_symbols(S, s, q, b, &at); m; m &= m - 1, ++at)
        ones |= ((S.col(at >> 5, b) >> (at & 31)) & 1u) << ctz32(m);
    return ones;
}

// finish: the column words of a propagation or cleanup stripe back into the bitmaps; returns the
// samples that turned significant
template <int L, int Q>
T1D_HD uint32_t stripe_finish_zc(const StripeState<L, Q>& S, int kind, int s, int q, int b, int cw) {
    if (8 * q >= cw) return 0;
    const uint32_t seen = S.cols(b)[q];  // the columns whose word holds visits (stripe_decode)
    uint32_t sg = 0, ng = 0, vs = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        if (Q == 1 && i >= cw) break;
        const uint32_t W = S.col(8 * q + i, b);
        sg |= gather4(W >> 4) << (4 * i);
        ng |= ((W >> 23) & 15u) << (4 * i);
        if (kind == kPassSP && ((seen >> i) & 1u)) vs |= gather4(W) << (4 * i);
    }
    const uint32_t ones = sg & ~S.sig(s, q, b);
    S.sig(s, q, b) = sg;
    S.neg(s, q, b) = ng & sg;
    if (kind == kPassSP) S.vis(s, q, b) = vs;
    return ones;
}

// bit p of the magnitudes of word q's samples `ones`.  A block's samples belong to one lane at a
// time; the atomic is a store that needs no load to return (its result is not read).
T1D_HD void stripe_add_bits(uint32_t ones, int32_t* blk, size_t pitch, int s, int q, int p) {
    while (ones) {
        const int i = ctz32(ones);
        ones &= ones - 1;
        int32_t* at = blk + (size_t)(4 * s + (i & 3)) * pitch + 8 * q + (i >> 2);
#ifdef __CUDA_ARCH__
        atomicOr(reinterpret_cast<unsigned int*>(at), 1u << p);
#else
        *at |= 1 << p;
#endif
    }
}

T1D_HD uint32_t float_bits(float f) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(f);
#else
    uint32_t u;
    memcpy(&u, &f, 4);
    return u;
#endif
}
T1D_HD float bits_float(uint32_t u) {
#ifdef __CUDA_ARCH__
    return __uint_as_float(u);
#else
    float f;
    memcpy(&f, &u, 4);
    return f;
#endif
}

// The MQ decoder (T.800 C.3).  A is kept as a float of the 16-bit register's value (integers below
// 2^16: exact), whose exponent is restored to renormalise, so that no leading-zero count is in the
// chain; C has its 16 compared bits on top.  The byte after the current one is loaded a byte-in ahead.
struct MqReg {
    const uint8_t* data;
    int len, bp, CT;
    float A;
    uint32_t C, B, n1;
    T1D_HD uint32_t byte(int i) const { return i < len ? data[i] : 0xFFu; }
    T1D_HD void bytein() {
        const bool ff = B == 0xFFu, end = ff && n1 > 0x8Fu;
        C += end ? 0xFF00u : n1 << (ff ? 9 : 8);
        CT = ff && !end ? 7 : 8;
        if (!end) {
            B = n1;
            ++bp;
            n1 = byte(bp + 1);
        }
    }
    T1D_HD void init(const uint8_t* d, int n) {
        data = d;
        len = n;
        bp = 0;
        B = byte(0);
        n1 = byte(1);
        C = B << 16;
        bytein();
        C <<= 7;
        CT -= 7;
        A = 32768.0f;
    }
    // one decision in a context of state e: the decision; *moved != 0 when the state changes, to
    // table entry *to
    T1D_HD uint32_t decide(MqdState e, uint32_t* moved, uint32_t* to) {
        constexpr uint32_t EXP = 0x47000000u;  // exponent field of 0x8000 <= A < 0x10000
        const uint32_t Q = e.y & 0xFFFF0000u;
        const float q = bits_float(e.x & 0x7FFFFFFFu), a1 = A - q;
        const bool lo = C < Q, lps = lo != (a1 < q);
        C -= lo ? 0u : Q;
        const uint32_t m = float_bits(lo ? q : a1);
        A = bits_float((m & 0x7FFFFFu) | EXP);
        *moved = EXP - (m & 0x7F800000u);
        *to = (e.y >> (lps ? 8 : 0)) & 0x7Fu;
        int sh = (int)(*moved >> 23);
        while (sh > CT) {  // the shifts up to the next byte, the byte, the rest
            C <<= CT;
            sh -= CT;
            bytein();
        }
        C <<= sh;
        CT -= sh;
        return (e.x >> 31) ^ (uint32_t)lps;
    }
};

// entry of the 94-entry state table (index = state * 2 + MPS)
__host__ __device__ inline MqdState stripe_mq_entry(int i) {
    const int st = i >> 1, mps = i & 1;
    const int sw = st == 0 || st == 6 || st == 14;
    return MqdState{float_bits((float)QE(st)) | ((uint32_t)mps << 31),
                    ((uint32_t)QE(st) << 16) | ((uint32_t)(NLPS(st) * 2 + (mps ^ sw)) << 8) |
                        (uint32_t)(NMPS(st) * 2 + mps)};
}

// Lookup tables of the stripe decoder.  sc is indexed by the column word's own bit layout: bits 1,
// 3, 5, 7 the significance above, left, right, below; bits 4, 0, 2, 6 their signs.
struct StripeTables {
    uint8_t zc[4][512];
    uint8_t sc[256];
    MqdState mq[94];
};
__host__ __device__ inline void fill_stripe_tables_entry(StripeTables& T, int i) {
    if (i < 4 * 512) {
        const int o = i >> 9, n = i & 511;
        const int h = ((n >> 3) & 1) + ((n >> 5) & 1), v = ((n >> 1) & 1) + ((n >> 7) & 1);
        const int d = (n & 1) + ((n >> 2) & 1) + ((n >> 6) & 1) + ((n >> 8) & 1);
        T.zc[o][n] = (uint8_t)zc_label_calc(o, h, v, d);
    }
    if (i < 256) {
        auto c = [&](int sg, int ng) { return ((i >> sg) & 1) ? (((i >> ng) & 1) ? -1 : 1) : 0; };
        int hc = max(-1, min(1, c(3, 0) + c(5, 2))), vc = max(-1, min(1, c(1, 4) + c(7, 6)));
        int xr = 0;
        if (hc < 0 || (hc == 0 && vc < 0)) { hc = -hc; vc = -vc; xr = 1; }
        T.sc[i] = (uint8_t)((hc == 0 ? (vc ? 10 : 9) : 12 + vc) | (xr << 7));
    }
    if (i < 94) T.mq[i] = stripe_mq_entry(i);
}

// What a lane's symbol loops touch: its block's column words and context states and the tables.  On
// the device 32-bit shared-memory addresses that the compiler cannot see through (it computes the
// address of a shared array anew for every access otherwise, special-register read included).
template <int L, int Q>
struct LaneMem {
#ifdef __CUDA_ARCH__
    uint32_t cols, ctxs, zcs, scs, mqs;
    __device__ __forceinline__ LaneMem(const StripeState<L, Q>& S, const StripeTables& T, int orient, int b)
        : cols(addr(&S.col(0, b))), ctxs(addr(&S.ctx(0, b))), zcs(addr(T.zc[orient])), scs(addr(T.sc)), mqs(addr(T.mq)) {
        asm volatile("" : "+r"(cols), "+r"(ctxs), "+r"(zcs), "+r"(scs), "+r"(mqs));
    }
    __device__ __forceinline__ static uint32_t addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
    __device__ __forceinline__ uint32_t col(int x) const {
        uint32_t v;
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(cols + x * (4 * L)) : "memory");
        return v;
    }
    __device__ __forceinline__ void col_set(int x, uint32_t v) const {
        asm volatile("st.shared.u32 [%0], %1;" ::"r"(cols + x * (4 * L)), "r"(v) : "memory");
    }
    __device__ __forceinline__ MqdState ctx(uint32_t k) const { return load(ctxs + k * (8 * L)); }
    __device__ __forceinline__ MqdState entry(uint32_t i) const { return load(mqs + 8 * i); }
    __device__ __forceinline__ void ctx_set_if(uint32_t cond, uint32_t k, MqdState v) const {
        asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %3, 0;\n @p st.shared.v2.u32 [%0], {%1, %2};\n}" ::"r"(
                         ctxs + k * (8 * L)),
                     "r"(v.x), "r"(v.y), "r"(cond)
                     : "memory");
    }
    __device__ __forceinline__ uint32_t zc(uint32_t i) const { return byte(zcs + i); }
    __device__ __forceinline__ uint32_t sc(uint32_t i) const { return byte(scs + i); }
    __device__ __forceinline__ static MqdState load(uint32_t at) {
        MqdState v;
        asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(at) : "memory");
        return v;
    }
    __device__ __forceinline__ static uint32_t byte(uint32_t at) {
        uint32_t v;
        asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(at) : "memory");
        return v;
    }
#else
    const StripeState<L, Q>& S;
    const StripeTables& T;
    int o, b;
    LaneMem(const StripeState<L, Q>& s, const StripeTables& t, int orient, int blk) : S(s), T(t), o(orient), b(blk) {}
    uint32_t col(int x) const { return S.col(x, b); }
    void col_set(int x, uint32_t v) const { S.col(x, b) = v; }
    MqdState ctx(uint32_t k) const { return S.ctx((int)k, b); }
    MqdState entry(uint32_t i) const { return T.mq[i]; }
    void ctx_set_if(uint32_t cond, uint32_t k, MqdState v) const {
        if (cond) S.ctx((int)k, b) = v;
    }
    uint32_t zc(uint32_t i) const { return T.zc[o][i]; }
    uint32_t sc(uint32_t i) const { return T.sc[i]; }
#endif
};

// One lane's block and its coder.
template <int L, int Q>
struct StripeLane {
    StripeState<L, Q> S;
    LaneMem<L, Q> mem;
    int b, cw, ch;
    MqReg m;
    RawD rd;
    bool raw;

    T1D_HD void reset_contexts() const {
        for (int k = 0; k < 19; ++k)
            S.ctx(k, b) = mem.entry(k == 0 ? 4 * 2 : (k == 17 ? 3 * 2 : (k == 18 ? 46 * 2 : 0)));
    }
    // one decision in context cx of state e; *up is the context's state after it where *moved
    template <bool STYLED>
    T1D_HD uint32_t dec(uint32_t cx, MqdState e, MqdState* up, uint32_t* moved) {
        *up = e;
        *moved = 0;
        if (STYLED && raw) return (uint32_t)rd.bit();
        uint32_t to;
        const uint32_t d = m.decide(e, moved, &to);
        *up = mem.entry(to);
        mem.ctx_set_if(*moved, cx, *up);
        return d;
    }
    template <bool STYLED>
    T1D_HD uint32_t dec(uint32_t cx) {
        MqdState up;
        uint32_t moved;
        return dec<STYLED>(cx, mem.ctx(cx), &up, &moved);
    }
    // the start of pass q of npasses: contexts and segments of a styled block
    template <bool STYLED>
    T1D_HD void begin(int q, int npasses, const uint8_t* data, int len, int style, const uint32_t* pe) {
        if (q == 0) reset_contexts();
        if (!STYLED) {
            if (q == 0) m.init(data, len);
            return;
        }
        if (q > 0 && (style & J2K_CBLK_RESET)) reset_contexts();
        raw = j2k_pass_raw(style, q);
        if (q == 0 || j2k_pass_terminated(style, q - 1, npasses)) {  // a new segment
            int e = q;
            while (!j2k_pass_terminated(style, e, npasses)) ++e;
            int b0 = q ? (int)min(pe[q - 1], (uint32_t)len) : 0;
            int b1 = (int)min(pe[e], (uint32_t)len);
            if (b1 < b0) b1 = b0;
            if (raw) rd.init(data + b0, b1 - b0);
            else m.init(data + b0, b1 - b0);
        }
    }

    // samples of a column that a pass codes, at 3k
    template <int KIND>
    T1D_HD static uint32_t candidates(uint32_t W, uint32_t rv) {
        const uint32_t c = ~(W >> 4) & rv;
        return KIND == kPassSP ? c & near_rows(W) : c & ~spread4((W >> 23) & 15u);
    }
    // run-length mode: four samples to code, no significant one around them
    template <int KIND>
    T1D_HD static bool run_length(uint32_t W, uint32_t c) {
        return KIND == kPassCU && c == 0x249u && !(W & 0x3FFFFu);
    }

    // Propagation (KIND kPassSP) or cleanup (kPassCU) symbols of a stripe, a zero-coding or run-length
    // decision a turn.  While it is decoded the symbol that follows a 0 is made ready (next row or
    // next column, its label and its context's state), which is most of a turn's latency; a 1 takes
    // the slow way: sign, column word, and the next symbol anew.
    template <bool STYLED, int KIND>
    T1D_HD void decode_zc(uint32_t rv) {
        uint32_t next_set = S.colset(1, b);
        const uint32_t wide_hi = cw >= 64 ? ~0u : (cw > 32 ? (1u << (cw - 32)) - 1u : 0u);
        uint32_t carry = 0;  // what the column before leaves to the next one
        for (int h = 0; h < (Q > 4 ? 2 : 1); ++h) {
            const int x0 = 32 * h;
            uint32_t set = h ? next_set : S.colset(0, b), all = set;
            const uint32_t wide = h ? wide_hi : (cw >= 32 ? ~0u : (1u << cw) - 1u);
            int x = h ? -1 : -2;
            uint32_t W = 0, c = 0, v = 0;
            // the next column that has a symbol (propagation: one reached by a carry may have none)
            const auto fetch = [&]() {
                do {
                    const int nx = ctz32(set);
                    set &= set - 1;
                    W = mem.col(x0 + nx) | (nx == x + 1 ? carry : 0u);
                    x = nx;
                    carry = 0;
                    c = candidates<KIND>(W, rv);
                    if (KIND == kPassSP && !c) mem.col_set(x0 + x, W & ~0x249u);
                } while (KIND == kPassSP && !c && set);
                v = 0;
            };
            const auto put = [&]() { mem.col_set(x0 + x, KIND == kPassSP ? (W & ~0x249u) | v : W); };
            if (set) fetch();
            if (c) {
                bool run = run_length<KIND>(W, c);
                int k3 = ctz32(c);
                uint32_t cx = run ? 17u : mem.zc((W >> k3) & 511u);
                MqdState e = mem.ctx(cx);
                for (;;) {
                    // the symbol after a 0: the column's next row, or the next column
                    const uint32_t c2 = run ? 0u : c & (c - 1);
                    const int nx = ctz32(set) & (Q > 4 ? 31 : 8 * Q - 1);
                    const uint32_t Wn = mem.col(x0 + nx) | (nx == x + 1 ? carry : 0u);
                    const uint32_t W2 = c2 ? W : Wn, d2 = c2 ? c2 : candidates<KIND>(Wn, rv);
                    const int k32 = ctz32(d2) & 15;
                    const bool run2 = !c2 && run_length<KIND>(Wn, d2);
                    const uint32_t cx2 = run2 ? 17u : mem.zc((W2 >> k32) & 511u);
                    MqdState e2 = mem.ctx(cx2);
                    MqdState up;
                    uint32_t moved;
                    uint32_t bit = dec<STYLED>(cx, e, &up, &moved);
                    if (KIND == kPassSP) v |= 1u << k3;
                    if (!bit) {
                        if (!c2) {
                            put();
                            if (!set) break;
                            if (KIND == kPassSP && !d2) {  // reached by a carry, without a sample to code
                                fetch();
                                if (!c) break;
                                k3 = ctz32(c);
                                cx = mem.zc((W >> k3) & 511u);
                                e = mem.ctx(cx);
                                continue;
                            }
                            x = nx;
                            set &= set - 1;
                            v = 0;
                            carry = 0;
                        }
                        const bool changed = cx2 == cx && moved != 0;
                        e.x = changed ? up.x : e2.x;
                        e.y = changed ? up.y : e2.y;
                        W = W2;
                        c = d2;
                        k3 = k32;
                        cx = cx2;
                        run = run2;
                        continue;
                    }
                    if (KIND == kPassCU && run) {  // the row of the first 1
                        uint32_t k = 0;
#pragma unroll 1
                        for (int i = 0; i < 2; ++i) k = 2 * k + dec<STYLED>(18u);
                        k3 = 3 * (int)k;
                    }
                    const int k = (k3 * 11) >> 5;
                    const uint32_t y = W >> k3, z = W >> (18 + k);
                    const uint32_t sc = mem.sc((y & 0xAAu) | (z & 0x51u) | ((z >> 8) & 4u));
                    uint32_t sg = dec<STYLED>(sc & 31u);
                    if (!(STYLED && raw)) sg ^= sc >> 7;
                    W |= (16u << k3) | (sg << (23 + k));
                    carry |= (8u << k3) | (sg << (18 + k));
                    if (KIND == kPassSP) {  // the next column has a candidate now
                        const uint32_t add = x < 31 ? (2u << x) & wide : 0u;
                        set |= add;
                        all |= add;
                        if (x == 31 && h == 0) next_set |= 1u & wide_hi;
                        c = candidates<KIND>(W, rv);
                    }
                    c &= 0x249u & (~1u << k3);  // rows below this one
                    run = false;
                    if (!c) {
                        put();
                        if (!set) break;
                        fetch();
                        if (!c) break;
                        run = run_length<KIND>(W, c);
                    }
                    k3 = ctz32(c);
                    cx = run ? 17u : mem.zc((W >> k3) & 511u);
                    e = mem.ctx(cx);
                }
            }
            if (KIND == kPassSP) S.colset(h, b) = all;
            if (x != 31) carry = 0;  // only column 31 is next to column 32
        }
    }

    // refinement symbols of a stripe, listed by stripe_prepare_mr; the context state of the next
    // symbol is loaded a symbol ahead
    template <bool STYLED>
    T1D_HD void decode_mr() {
        const int n = (int)S.colset(0, b);
        uint32_t out = 0;
        if (STYLED && raw) {
            for (int i = 0; i < n; ++i) {
                out |= (uint32_t)rd.bit() << (i & 31);
                if ((i & 31) == 31 || i == n - 1) mem.col_set(i >> 5, out), out = 0;
            }
            return;
        }
        if (n == 0) return;
        uint32_t labels = mem.col(0), cx = labels & 31u;
        MqdState e = mem.ctx(cx);
        for (int i = 0; i < n; ++i) {
            labels >>= 8;
            if ((i & 3) == 3) labels = mem.col(((i + 1) >> 2) & (8 * Q - 1));
            const uint32_t ncx = min(labels & 31u, 18u);  // (past the last label: any context)
            const MqdState ne = mem.ctx(ncx);
            MqdState up;
            uint32_t moved;
            out |= dec<false>(cx, e, &up, &moved) << (i & 31);
            const bool changed = ncx == cx && moved != 0;
            e.x = changed ? up.x : ne.x;
            e.y = changed ? up.y : ne.y;
            cx = ncx;
            if ((i & 31) == 31) mem.col_set(i >> 5, out), out = 0;
        }
        if (n & 31) mem.col_set(n >> 5, out);
    }
};

// valid rows of stripe s of a block of ch rows, at 3k
T1D_HD uint32_t stripe_rows(int ch, int s) {
    const int n = ch - 4 * s;
    return n >= 4 ? 0x249u : 0x249u & ((1u << (3 * n)) - 1u);
}
