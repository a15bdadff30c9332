// The MQ encoder of one lane (T.800 C.2), in two parts that meet every eight symbols.
//
// Interval part.  A, Qe and the comparisons of the conditional exchange are kept as floats: A is
// the float whose value is the 16-bit register (0x8000 <= A < 0x10000, so its exponent field is
// constant), which makes the renormalisation one bit operation -- put the exponent field back --
// and the number of shifts the difference of two exponent fields.  All values are integers below
// 2^16, so every float operation is exact.  With s = +1 when the decision is the MPS and -1 when
// it is the LPS, T.800's four cases are one maximum:
//     m = max(s * (A - Qe), s * Qe),   new A = |m|,   Qe is added to C iff m is the first operand
// (an MPS keeps the larger part of the interval, an LPS the smaller one; of equal parts the MPS
// takes the first and the LPS the second, which the comparison with a half less than Qe decides).
// The sign rides along in Qe's sign bit.  The chain from symbol to symbol is then three
// operations: restore the exponent, multiply-add, maximum.
//
// Code part.  The eight pairs (value added to C, shifts) of a group are folded into C in one go, and
// the bytes that became due are taken from a 64-bit C afterwards.  A byte taken late already holds
// the carry of the additions after it, which T.800 would add to it one byte later; the result is
// the same unless the byte was 0xFF when it was due (then the carry stays in the next byte's stuffed
// bit).  That byte reads as 0 with a carry out of it, so whenever one may be such a byte, or the
// shifts are too many, the group is coded again byte by byte in T.800's order.
//
// Host-callable: the same code runs on the CPU in the tests.

#define MQ_HD __host__ __device__ __forceinline__

// Context state: x = Qe as a float, the MPS in the sign bit; y = Qe | entry after an MPS << 16 |
// entry after an LPS << 24 (entries of the 94-entry table, state * 2 + MPS).
struct alignas(8) MqState {
    uint32_t x, y;
};

MQ_HD uint32_t mq_bits(float f) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(f);
#else
    uint32_t u;
    memcpy(&u, &f, 4);
    return u;
#endif
}
MQ_HD float mq_float(uint32_t u) {
#ifdef __CUDA_ARCH__
    return __uint_as_float(u);
#else
    float f;
    memcpy(&f, &u, 4);
    return f;
#endif
}

constexpr uint32_t kMqExp = 0x47000000u;  // exponent field of 0x8000 <= A < 0x10000

struct MqCoder {
    float A;
    uint32_t C, B;   // B: the last byte made, which may still receive a carry
    int CT, cnt;     // cnt: bytes made, B included
    uint32_t wacc;   // the last four bytes before B, oldest lowest
    uint32_t* out;   // word-aligned codeword buffer
    int cap;         // bytes
    bool ovf;

    MQ_HD void init(uint32_t* o, int bytes) {
        A = 32768.0f;
        C = 0;
        B = 0;
        CT = 12;
        cnt = 0;
        wacc = 0;
        out = o;
        cap = bytes;
        ovf = false;
    }
    // B is final: into the word, which is stored when complete (before the first byte B is none)
    MQ_HD void push() {
        wacc = (wacc >> 8) | (B << 24);
        if (cnt != 0 && (cnt & 3) == 0) {
            if (cnt <= cap) out[(cnt >> 2) - 1] = wacc;
            else ovf = true;
        }
    }
    // T.800 BYTEOUT
    MQ_HD void byteout() {
        const bool carry = B != 0xFFu && (C >> 27) != 0;
        B += carry ? 1u : 0u;
        C &= carry ? 0x7FFFFFFu : ~0u;
        const bool ff = B == 0xFFu;
        push();
        ++cnt;
        B = (C >> (ff ? 20 : 19)) & 0xFFu;
        C &= ff ? 0xFFFFFu : 0x7FFFFu;
        CT = ff ? 7 : 8;
    }
    MQ_HD void shift(int sh) {
        while (sh >= CT) {
            C <<= CT;
            sh -= CT;
            byteout();
        }
        C <<= sh;
        CT -= sh;
    }
    // interval part of one symbol in state e: the decision in bit 31 of d31, the value added to C
    // in *add; returns the shift count << 23.  *next: table entry of the state after a shift.
    // *width: the new A before the shifts, with either sign (the state changes iff it is below 0x8000).
    MQ_HD uint32_t interval(MqState e, uint32_t d31, uint32_t* add, uint32_t* next, float* width) {
        const uint32_t qs = e.x ^ (d31 & 0x80000000u);
        const float q = mq_float(qs), s = mq_float((qs & 0x80000000u) | 0x3F800000u);
#ifdef __CUDA_ARCH__
        const float a1 = __fmaf_rn(A, s, -q), low = __fmaf_rn(s, -0.5f, q);
        const uint32_t m = mq_bits(fmaxf(a1, q));
        *next = __byte_perm(e.y, 0u, 0x4442u + (qs >> 31));
#else
        const float a1 = A * s - q, low = q - 0.5f * s;
        const uint32_t m = mq_bits(a1 > q ? a1 : q);
        *next = (e.y >> ((qs >> 31) ? 24 : 16)) & 0xFFu;
#endif
        *add = a1 > low ? e.y & 0xFFFFu : 0u;
        A = mq_float((m & 0x7FFFFFu) | kMqExp);
        *width = mq_float(m);
        return kMqExp - (m & 0x7F800000u);
    }
    // Takes the bytes out of c, a C that has been shifted -ct times since the first of them was due;
    // false, with everything as it was, when a byte read late may have been 0xFF when it was due.
    MQ_HD bool bytes_late(uint64_t c, int ct) {
        const uint32_t B0 = B, w0 = wacc;
        const int cnt0 = cnt;
        const bool ovf0 = ovf;
        bool doubt = (c >> (28 - ct)) != 0, again = false;
        // the due byte at bits 62..55, its carry at 63 (each byte taken moves the next one up)
        uint64_t t = c << (36 + ct);
        do {
            const uint32_t top = (uint32_t)(t >> 32);
            const bool carry = B != 0xFFu && (top >> 31) != 0;
            B += carry ? 1u : 0u;
            const bool ff = B == 0xFFu;
            const uint32_t v = ((carry ? top & 0x7FFFFFFFu : top) >> (ff ? 24 : 23)) & 0xFFu;
            // a 0 that a carry came out of, into B now or into the byte taken before it
            doubt |= v == 0 && (carry || again);
            push();
            ++cnt;
            B = v;
            t = (t << (ff ? 8 : 9)) >> 1;
            ct += ff ? 7 : 8;
            again = true;
        } while (ct <= 0);
        if (doubt) {
            B = B0;
            wacc = w0;
            cnt = cnt0;
            ovf = ovf0;
            return false;
        }
        C = (uint32_t)(t >> (36 + ct));
        CT = ct;
        return true;
    }
    // code part of eight symbols, each an addition | shifts << 16; each half's additions are summed
    // by themselves (32 bits hold them up to 15 shifts) before C comes in.  False where the symbols
    // have to be coded one by one.
    MQ_HD bool code8(const uint32_t (&e)[8]) {
        uint32_t P[2] = {0, 0};
        int S[2] = {0, 0};
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
        for (int j = 0; j < 4; ++j)
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
            for (int h = 0; h < 2; ++h) {
                const uint32_t v = e[4 * h + j];
                P[h] = (P[h] + (v & 0xFFFFu)) << (v >> 16);
                S[h] += (int)(v >> 16);
            }
        const int both = S[0] + S[1];
        if (both < CT) {
            C = (((C << S[0]) + P[0]) << S[1]) + P[1];
            CT -= both;
            return true;
        }
        if (S[0] > 15 || S[1] > 15) return false;
        return bytes_late(((uint64_t)C << both) + ((uint64_t)P[0] << S[1]) + P[1], CT - both);
    }
    // the same one by one
    MQ_HD void code_each(const uint32_t (&e)[8]) {
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
        for (int j = 0; j < 8; ++j) {
            C += e[j] & 0xFFFFu;
            shift((int)(e[j] >> 16));
        }
    }
    // FLUSH (C.2.9); a last byte of 0xFF is dropped.  Returns the codeword's length.
    MQ_HD int flush() {
        const uint32_t a = ((mq_bits(A) & 0x7FFFFFu) | 0x800000u) >> 8;
        const uint32_t top = C + a;
        C |= 0xFFFFu;
        if (C >= top) C -= 0x8000u;
        C <<= CT;
        byteout();
        C <<= CT;
        byteout();
        push();
        uint8_t* tail = reinterpret_cast<uint8_t*>(out);
        const int r = cnt & 3;
        for (int k = 0; k < r; ++k) {
            if (cnt - r + k < cap) tail[cnt - r + k] = (uint8_t)(wacc >> (8 * (4 - r + k)));
            else ovf = true;
        }
        return cnt - (B == 0xFFu ? 1 : 0);
    }
};

#ifdef __CUDA_ARCH__
#define MQ_LOAD16(p) __ldcs(p)
#else
#define MQ_LOAD16(p) (*(p))
#endif

// One lane's 32 context states, 8 << SHIFT bytes apart, and the state table.  On the device both
// are 32-bit shared-memory addresses that the compiler cannot see through: it computes the address
// of a shared array anew for every access otherwise, with a special-register read in it.
// COPIES: the table holds each entry that many times side by side, and lane l reads copy l % COPIES
// (the lanes' entries then fall in distinct banks but for pairs of them).
template <int SHIFT, int COPIES = 1>
struct MqMem {
#ifdef __CUDA_ARCH__
    uint32_t st, tab;
    __device__ __forceinline__ MqMem(MqState* s, const MqState* t)
        : st((uint32_t)__cvta_generic_to_shared(s)), tab((uint32_t)__cvta_generic_to_shared(t)) {
        asm volatile("" : "+r"(st), "+r"(tab));
    }
    // cx8: the context << (SHIFT + 3)
    __device__ __forceinline__ MqState state(uint32_t cx8) const { return load(st + cx8); }
    __device__ __forceinline__ MqState entry(uint32_t i) const { return load(tab + 8 * COPIES * i); }
    // stores v when |width| is below 0x8000 (compared as it comes out of the maximum: the shift count
    // takes three operations more)
    __device__ __forceinline__ void store_if_below(float width, uint32_t cx8, MqState v) const {
        asm volatile("{\n .reg .pred p;\n .reg .f32 t;\n abs.f32 t, %3;\n setp.lt.f32 p, t, 0f47000000;\n"
                     " @p st.shared.v2.u32 [%0], {%1, %2};\n}" ::"r"(st + cx8),
                     "r"(v.x), "r"(v.y), "f"(width)
                     : "memory");
    }
    __device__ __forceinline__ static MqState load(uint32_t at) {
        MqState v;
        asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(at) : "memory");
        return v;
    }
#else
    MqState* st;
    const MqState* tab;
    MqMem(MqState* s, const MqState* t) : st(s), tab(t) {}
    MqState state(uint32_t cx8) const { return st[cx8 / 8]; }
    MqState entry(uint32_t i) const { return tab[COPIES * i]; }
    void store_if_below(float width, uint32_t cx8, MqState v) const {
        if (fabsf(width) < 32768.0f) st[cx8 / 8] = v;
    }
#endif
    // byte j of a symbol word as cx8 (j = 4: the first byte of the next word)
    MQ_HD static uint32_t context(uint32_t w, int j) {
        const int left = SHIFT + 3 - 8 * j;
        return (left >= 0 ? w << left : w >> -left) & (31u << (SHIFT + 3));
    }
};

// The interval part's walk over a symbol stream: n symbols at syms (16-byte aligned; bits 0-4
// context, bit 7 decision) in 16-byte chunks, two in flight; the state of the next symbol's context
// is loaded a symbol ahead and replaced when this symbol changes the same context.
template <class Mem>
struct MqSymbols {
    const Mem mem;
    const uint4* sp;
    int n, nchunks;
    uint4 c0, c1;
    uint32_t cx;
    MqState cur;
    MQ_HD MqSymbols(const uint8_t* syms, int count, Mem m)
        : mem(m), sp(reinterpret_cast<const uint4*>(syms)), n(count), nchunks((count + 15) >> 4) {
        const uint4 z = make_uint4(0, 0, 0, 0);
        c0 = nchunks > 0 ? MQ_LOAD16(sp) : z;
        c1 = nchunks > 1 ? MQ_LOAD16(sp + 1) : z;
        cx = mem.context(c0.x, 0);
        cur = mem.state(cx);
    }
    // chunk k (in order), then the one after it in c0
    MQ_HD uint4 next(int k) {
        const uint4 w = c0;
        c0 = c1;
        c1 = k + 2 < nchunks ? MQ_LOAD16(sp + k + 2) : make_uint4(0, 0, 0, 0);
        return w;
    }
    // four symbols w, of which `left` exist, the next one in wnext: put(j, value added to C, shifts
    // << 23); without branches, so that the chains of neighbouring symbols overlap
    template <class Put>
    MQ_HD void group(MqCoder& e, uint32_t w, uint32_t wnext, int left, Put put) {
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
        for (int j = 0; j < 4; ++j) {
            if (j > 0 && j >= left) {
                put(j, 0u, 0u);
                continue;
            }
            const uint32_t ncx = j < 3 ? mem.context(w, j + 1) : mem.context(wnext, 0);
            const MqState nx = mem.state(ncx);
            uint32_t to, add;
            float width;
            const uint32_t moved = e.interval(cur, w << (24 - 8 * j), &add, &to, &width);
            put(j, add, moved);
            const MqState up = mem.entry(to);
            mem.store_if_below(width, cx, up);
            // the next symbol's state: the one loaded ahead, unless this symbol has changed it
            const bool changed = ncx == cx && fabsf(width) < 32768.0f;
            cur = MqState{changed ? up.x : nx.x, changed ? up.y : nx.y};
            cx = ncx;
        }
    }
};

// Both parts by one lane
template <class Mem>
MQ_HD void mq_encode(MqCoder& e, const uint8_t* syms, int n, Mem mem) {
    MqSymbols<Mem> src(syms, n, mem);
    for (int k = 0; k < src.nchunks; ++k) {
        const uint4 c = src.next(k);
        uint32_t wa = c.x, wb = c.y, wc = c.z, wd = c.w, ev[8];
        const auto put = [&](int j, uint32_t add, uint32_t moved) { ev[j] = add | (moved >> 7); };
        const auto put4 = [&](int j, uint32_t add, uint32_t moved) { ev[4 + j] = add | (moved >> 7); };
#ifdef __CUDA_ARCH__
#pragma unroll 1
#endif
        for (int i = 16 * k; i < 16 * k + 16 && i < n; i += 8) {
            if (n - i >= 8) {
                src.group(e, wa, wb, 4, put);
                src.group(e, wb, wc, 4, put4);
            } else {
                ev[4] = ev[5] = ev[6] = ev[7] = 0;
                src.group(e, wa, wb, n - i, put);
                if (n - i > 4) src.group(e, wb, wc, n - i - 4, put4);
            }
            if (!e.code8(ev)) e.code_each(ev);
            wa = wc;
            wb = wd;
            wc = src.c0.x;
        }
    }
}

MQ_HD MqState mq_table_entry(uint32_t qe, uint32_t nmps, uint32_t nlps, uint32_t sw, uint32_t mps) {
    return MqState{mq_bits((float)qe) | (mps << 31),
                   qe | ((nmps * 2 + mps) << 16) | ((nlps * 2 + (mps ^ sw)) << 24)};
}
