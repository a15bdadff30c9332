// EBCOT tier-1 decoder (T.800 Annex D context modelling + Annex C.3 MQ decoder).
//
// The reference has no decoder for this stage (src/OCLDecoder.cpp:35-38 runs only the "reverse"
// DWT).  Decoding is serial per code-block: every context depends on the bits decoded before it.
// The kernel runs one code-block per lane, 1 to 16 in a warp, and takes all
// work that is not a block's own serial chain out of the lanes' loops (t1dec_stripe.cuh).  What
// bounds it: the chain of dependent instructions per symbol (about 91 warp instructions and 360
// cycles a symbol with one block per warp), and with 4 blocks per warp the ALU pipe, since the lanes
// are at different kinds of symbols (1.74 times the instructions of one).  Round trips host to host
// on B200, against a decoder whose lanes kept 64-bit row masks and gathered each column's
// neighbourhood themselves: 512 x 512 gray 15.3 -> 5.5 ms, 2048 x 2048 colour 18.8 -> 10.5 ms,
// 4096 x 4096 colour 28.5 -> 20.5 ms.
// The warp clears its blocks' output regions first and applies the signs at the end; magnitude bits
// go to the output plane by fire-and-forget atomic ORs (each block owns its region).
#include <atomic>
#include <cstring>

#include <cub/cub.cuh>

#include "j2k_internal.cuh"

namespace {

// T.800 Table C.2 (probability estimation), device and host copies
__constant__ uint16_t d_qe[47] = {
    0x5601, 0x3401, 0x1801, 0x0AC1, 0x0521, 0x0221, 0x5601, 0x5401, 0x4801, 0x3801, 0x3001, 0x2401,
    0x1C01, 0x1601, 0x5601, 0x5401, 0x5101, 0x4801, 0x3801, 0x3401, 0x3001, 0x2801, 0x2401, 0x2201,
    0x1C01, 0x1801, 0x1601, 0x1401, 0x1201, 0x1101, 0x0AC1, 0x09C1, 0x08A1, 0x0521, 0x0441, 0x02A1,
    0x0221, 0x0141, 0x0111, 0x0085, 0x0049, 0x0025, 0x0015, 0x0009, 0x0005, 0x0001, 0x5601};
__constant__ uint8_t d_nmps[47] = {
    1,  2,  3,  4,  5,  38, 7,  8,  9,  10, 11, 12, 13, 29, 15, 16, 17, 18, 19, 20, 21, 22, 23, 24,
    25, 26, 27, 28, 29, 30, 31, 32, 33, 34, 35, 36, 37, 38, 39, 40, 41, 42, 43, 44, 45, 45, 46};
__constant__ uint8_t d_nlps[47] = {
    1,  6,  9,  12, 29, 33, 6,  14, 14, 14, 17, 18, 20, 21, 14, 14, 15, 16, 17, 18, 19, 19, 20, 21,
    22, 23, 24, 25, 26, 27, 28, 29, 30, 31, 32, 33, 34, 35, 36, 37, 38, 39, 40, 41, 42, 43, 46};
[[maybe_unused]] static const uint16_t h_qe[47] = {
    0x5601, 0x3401, 0x1801, 0x0AC1, 0x0521, 0x0221, 0x5601, 0x5401, 0x4801, 0x3801, 0x3001, 0x2401,
    0x1C01, 0x1601, 0x5601, 0x5401, 0x5101, 0x4801, 0x3801, 0x3401, 0x3001, 0x2801, 0x2401, 0x2201,
    0x1C01, 0x1801, 0x1601, 0x1401, 0x1201, 0x1101, 0x0AC1, 0x09C1, 0x08A1, 0x0521, 0x0441, 0x02A1,
    0x0221, 0x0141, 0x0111, 0x0085, 0x0049, 0x0025, 0x0015, 0x0009, 0x0005, 0x0001, 0x5601};
[[maybe_unused]] static const uint8_t h_nmps[47] = {
    1,  2,  3,  4,  5,  38, 7,  8,  9,  10, 11, 12, 13, 29, 15, 16, 17, 18, 19, 20, 21, 22, 23, 24,
    25, 26, 27, 28, 29, 30, 31, 32, 33, 34, 35, 36, 37, 38, 39, 40, 41, 42, 43, 44, 45, 45, 46};
[[maybe_unused]] static const uint8_t h_nlps[47] = {
    1,  6,  9,  12, 29, 33, 6,  14, 14, 14, 17, 18, 20, 21, 14, 14, 15, 16, 17, 18, 19, 19, 20, 21,
    22, 23, 24, 25, 26, 27, 28, 29, 30, 31, 32, 33, 34, 35, 36, 37, 38, 39, 40, 41, 42, 43, 46};
#ifdef __CUDA_ARCH__
#define QE(i) d_qe[i]
#define NMPS(i) d_nmps[i]
#define NLPS(i) d_nlps[i]
#else
#define QE(i) h_qe[i]
#define NMPS(i) h_nmps[i]
#define NLPS(i) h_nlps[i]
#endif

__host__ __device__ __forceinline__ int zc_label_calc(int orient, int h, int v, int d) {
    if (orient == J2K_BAND_HH) {
        int hv = h + v;
        if (d >= 3) return 8;
        if (d == 2) return hv >= 1 ? 7 : 6;
        if (d == 1) return hv >= 2 ? 5 : (hv == 1 ? 4 : 3);
        return hv >= 2 ? 2 : (hv == 1 ? 1 : 0);
    }
    if (orient == J2K_BAND_HL) { int t = h; h = v; v = t; }
    if (h == 2) return 8;
    if (h == 1) return v >= 1 ? 7 : (d >= 1 ? 6 : 5);
    if (v == 2) return 4;
    if (v == 1) return 3;
    return d >= 2 ? 2 : d;
}

// Lookup tables shared by the warps of a CTA (the host path builds its own copy).
//   zc[o][n9]: zero-coding label for orientation o and the 9-bit significance neighbourhood n9
//              (bits 0-2: row above, columns x-1..x+1; 3-5: own row; 6-8: row below; the
//              sample's own bit 4 is ignored; a significant neighbour is n9 & 0x1EF != 0)
//   sc[n8]:    sign-coding label | xor bit << 7 for n8 = sigL negL sigR negR sigU negU sigD negD
//   mq[i]:     Qe | NMPS << 16 | NLPS << 22 | SWITCH << 28 of probability state i (Table C.2)
struct DecTables {
    uint8_t zc[4][512];
    uint8_t sc[256];
    uint32_t mq[47];
};

__host__ __device__ inline void fill_tables_entry(DecTables& T, int i) {
    if (i < 4 * 512) {
        const int o = i >> 9, n = i & 511;
        const int h = ((n >> 3) & 1) + ((n >> 5) & 1), v = ((n >> 1) & 1) + ((n >> 7) & 1);
        const int d = (n & 1) + ((n >> 2) & 1) + ((n >> 6) & 1) + ((n >> 8) & 1);
        T.zc[o][n] = (uint8_t)zc_label_calc(o, h, v, d);
    }
    if (i < 256) {
        auto c = [&](int sh) { return ((i >> sh) & 1) ? (((i >> (sh + 1)) & 1) ? -1 : 1) : 0; };
        int hc = max(-1, min(1, c(0) + c(2))), vc = max(-1, min(1, c(4) + c(6)));
        int xr = 0;
        if (hc < 0 || (hc == 0 && vc < 0)) { hc = -hc; vc = -vc; xr = 1; }
        T.sc[i] = (uint8_t)((hc == 0 ? (vc ? 10 : 9) : 12 + vc) | (xr << 7));
    }
    if (i < 47)
        T.mq[i] = (uint32_t)QE(i) | ((uint32_t)NMPS(i) << 16) | ((uint32_t)NLPS(i) << 22) |
                  ((uint32_t)(i == 0 || i == 6 || i == 14) << 28);
}

__host__ __device__ __forceinline__ int clz32(uint32_t v) {
#ifdef __CUDA_ARCH__
    return __clz(v);
#else
    return v ? __builtin_clz(v) : 32;
#endif
}

// Decoder state of one code-block: rows of 64-bit masks (row r + 1 holds block row r; rows 0
// and 65 are the zero border) and the 19 MQ context states.
struct DecSmem {
    uint64_t sig_[66], neg_[66], ref_[66], vis_[66];
    uint8_t st_[19];
    __host__ __device__ uint64_t& sig(int r) { return sig_[r]; }
    __host__ __device__ uint64_t& neg(int r) { return neg_[r]; }
    __host__ __device__ uint64_t& ref(int r) { return ref_[r]; }
    __host__ __device__ uint64_t& vis(int r) { return vis_[r]; }
    __host__ __device__ uint8_t& st(int k) { return st_[k]; }
};

// The same state for the lanes of a warp that decode L blocks side by side: word (a, r, lane) of
// mask array a at base[(a * 66 + r) * L + lane], context state k at stb[k * L + lane].
template <int L>
struct LaneState {
    uint64_t* base;
    uint8_t* stb;
    int lane;
    __device__ uint64_t& sig(int r) { return base[(0 * 66 + r) * L + lane]; }
    __device__ uint64_t& neg(int r) { return base[(1 * 66 + r) * L + lane]; }
    __device__ uint64_t& ref(int r) { return base[(2 * 66 + r) * L + lane]; }
    __device__ uint64_t& vis(int r) { return base[(3 * 66 + r) * L + lane]; }
    __device__ uint8_t& st(int k) { return stb[k * L + lane]; }
};
template <int L>
__host__ __device__ constexpr size_t lane_state_bytes() {  // one warp's share: the masks, then the context states
    return (size_t)4 * 66 * L * 8 + (((size_t)19 * L + 15) & ~(size_t)15);
}

struct Mqd {
    const uint8_t* data;
    int len, bp, CT;
    uint32_t A, C;
    __host__ __device__ uint32_t byte(int i) const { return i < len ? data[i] : 0xFFu; }
    __host__ __device__ void bytein() {
        if (byte(bp) == 0xFF) {
            if (byte(bp + 1) > 0x8F) {
                C += 0xFF00;
                CT = 8;
            } else {
                ++bp;
                C += byte(bp) << 9;
                CT = 7;
            }
        } else {
            ++bp;
            C += byte(bp) << 8;
            CT = 8;
        }
    }
    __host__ __device__ void init(const uint8_t* d, int n) {
        data = d;
        len = n;
        bp = 0;
        C = byte(0) << 16;
        bytein();
        C <<= 7;
        CT -= 7;
        A = 0x8000;
    }
    // renormalisation by the leading-zero count at once, stopping for a byte-in whenever CT
    // runs out (the same steps as the bit-by-bit loop of C.3.3)
    __host__ __device__ __forceinline__ void renorm() {
        int sh = clz32(A) - 16;
        while (sh > 0) {
            if (CT == 0) bytein();
            const int k = min(sh, CT);
            A <<= k;
            C <<= k;
            CT -= k;
            sh -= k;
        }
    }
    __host__ __device__ int decode(uint8_t& st, const uint32_t* mq) {
        const uint32_t sv = st;
        const uint32_t e = mq[sv >> 1];
        const uint32_t qe = e & 0xFFFF;
        const int mps = sv & 1;
        A -= qe;
        int D, nm = mps;
        uint32_t nidx;
        if ((C >> 16) >= qe) {
            C -= qe << 16;
            if (A & 0x8000) return mps;  // MPS, no renormalisation
            if (A < qe) {                // conditional exchange: LPS
                D = 1 - mps;
                nm ^= (int)(e >> 28);
                nidx = (e >> 22) & 63;
            } else {
                D = mps;
                nidx = (e >> 16) & 63;
            }
        } else {
            if (A < qe) {  // conditional exchange: MPS
                D = mps;
                nidx = (e >> 16) & 63;
            } else {
                D = 1 - mps;
                nm ^= (int)(e >> 28);
                nidx = (e >> 22) & 63;
            }
            A = qe;
        }
        st = (uint8_t)((nidx << 1) | nm);
        renorm();
        return D;
    }
};

// bits x-1, x, x+1 of a row mask (bit 0 = column x-1); columns outside 0..63 read as 0
__host__ __device__ __forceinline__ int ctz64(uint64_t v) {
#ifdef __CUDA_ARCH__
    return __ffsll((long long)v) - 1;
#else
    return __builtin_ctzll(v);
#endif
}
__host__ __device__ __forceinline__ uint32_t nb3(uint64_t m, int x) {
    return (uint32_t)(x > 0 ? (m >> (x - 1)) & 7 : (m << 1) & 7);
}

// sign-coding neighbourhood of stripe row k of a column whose significance / sign neighbourhoods
// are W / NW (bits 3r..3r+2: columns x-1..x+1 of window row r): sigL negL sigR negR sigU negU
// sigD negD
__host__ __device__ __forceinline__ uint32_t sign_nbhd(uint32_t W, uint32_t NW, int k) {
    const int b = 3 * k;
    return ((W >> (b + 3)) & 1) | (((NW >> (b + 3)) & 1) << 1) | (((W >> (b + 5)) & 1) << 2) |
           (((NW >> (b + 5)) & 1) << 3) | (((W >> (b + 1)) & 1) << 4) | (((NW >> (b + 1)) & 1) << 5) |
           (((W >> (b + 7)) & 1) << 6) | (((NW >> (b + 7)) & 1) << 7);
}

// Raw (bypass) segment reader, T.800 D.6: bits most significant first; a byte after 0xFF holds
// 7 bits (its top bit is a stuffed 0); past the end of the segment 0xFF is read.
struct RawD {
    const uint8_t* data;
    int len, pos, ct;
    uint32_t c;
    bool lastff;
    __host__ __device__ void init(const uint8_t* d, int n) {
        data = d;
        len = n;
        pos = 0;
        ct = 0;
        c = 0;
        lastff = false;
    }
    __host__ __device__ int bit() {
        if (ct == 0) {
            const uint32_t b = pos < len ? data[pos] : 0xFFu;
            ++pos;
            ct = lastff ? 7 : 8;
            lastff = b == 0xFF;
            c = b;
        }
        --ct;
        return (int)((c >> ct) & 1);
    }
};

#include "t1dec_stripe.cuh"

// the checks a decoder kernel makes of a job before touching its region
__device__ __forceinline__ bool dec_job_ok(const j2k_cb_job& J, const j2k_cb_desc& D, bool styled) {
    return !(J.cw == 0 || J.ch == 0 || J.cw > 64 || J.ch > 64 || J.orient > 3 || D.numbps > 31 ||
             D.npasses > 3 * D.numbps || D.length < 0 || (styled && D.npasses > J2K_PASS_STRIDE - 1));
}

// magnitude offset of a block cut at the end of a bit-plane above the last one (rate control):
// significant magnitudes are reconstructed at the middle of the interval their undecoded bits leave
__host__ __device__ __forceinline__ int32_t cut_half(int numbps, int npasses) {
    if (npasses < 3 * numbps - 2 && (npasses - 1) % 3 == 0) {
        const int plast = numbps - 1 - (npasses - 1) / 3;
        return plast > 0 ? 1 << (plast - 1) : 0;
    }
    return 0;
}

// Warps per CTA of the stripe decoder for L blocks per warp of Q words a stripe: with 4 or 8 blocks of
// 8 words one CTA's state fills an SM's shared memory (84 or 88 blocks; the 12288 blocks of a
// 4096 x 4096 colour image are then resident at once on 148 SMs).
template <int L, int Q>
__host__ __device__ constexpr int stripe_warps() {
    return Q == 1 ? 24 : L == 1 ? 16 : (L == 2 ? 20 : (L == 4 ? 21 : (L == 8 ? 11 : 5)));
}
constexpr size_t kStripeTablesBytes = (sizeof(StripeTables) + 15) & ~(size_t)15;
template <int L, int Q>
__host__ __device__ constexpr size_t stripe_smem_bytes(int warps) {
    return kStripeTablesBytes + (size_t)warps * stripe_state_words<L, Q>() * 4;
}

// L code-blocks per warp, one per lane, of at most 8 * Q columns (t1dec_stripe.cuh).  Groups of L consecutive blocks of
// `order` (longest codewords first) go to the warps of all CTAs in turn, then from a queue.  Blocks
// of more than half the longest codeword (keys: the lengths in that order) get a warp of their own,
// at most `alone` of them: a block runs fastest alone, and the others end before it anyway.
template <bool STYLED, int L, int Q>
__global__ void __launch_bounds__(32 * stripe_warps<L, Q>(), 1)
t1_decode_stripe_kernel(const j2k_cb_desc* __restrict__ descs, const uint8_t* __restrict__ bytes,
                        const j2k_cb_job* __restrict__ jobs, int njobs, int32_t* __restrict__ coeff,
                        uint32_t* __restrict__ err, int style, const uint32_t* __restrict__ pass_ends,
                        const uint8_t* __restrict__ job_style, const uint32_t* __restrict__ order,
                        const uint32_t* __restrict__ keys, int alone, uint32_t* __restrict__ queue) {
    extern __shared__ __align__(16) uint8_t dsm[];
    StripeTables& tabs = *reinterpret_cast<StripeTables*>(dsm);
    for (int i = threadIdx.x; i < 4 * 512; i += blockDim.x) fill_stripe_tables_entry(tabs, i);
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const StripeState<L, Q> S{reinterpret_cast<uint32_t*>(dsm + kStripeTablesBytes) + wid * stripe_state_words<L, Q>()};
    constexpr int R = (Q * L + 31) / 32;  // rounds of 32 (block, word) items per stripe
    constexpr int WX = Q == 1 ? 8 : 32, WY = 32 / WX;  // columns and rows of a block that the warp takes at a time
    if (L > 1 && alone > 0) {  // the number of leading keys above half the first one
        const uint32_t half = keys[0] / 2;
        int lo = 0, hi = alone;  // it is in lo..hi
        while (lo < hi) {
            const int step = (hi - lo + 31) / 32, at = lo + lane * step;  // keys[lo], keys[lo + step], ...
            const unsigned above = __ballot_sync(~0u, at < hi && keys[at] > half);
            const int n = __popc(above);  // (a run of ones from bit 0: the keys fall)
            if (n == 0) break;
            const int last = lo + (n - 1) * step;  // above half; the next probe is not
            hi = min(hi, last + step);
            lo = last + 1;
        }
        alone = lo;
    }
    const int ngroups = alone + (njobs - alone + L - 1) / L;
    for (int g = wid * (int)gridDim.x + (int)blockIdx.x; g < ngroups;) {
        const int j0 = g < alone ? g : alone + (g - alone) * L, nb = g < alone ? 1 : min(L, njobs - j0);
        j2k_cb_job J{};
        j2k_cb_desc D{};
        bool ok = false;
        const int jid = lane < nb ? (order ? (int)order[j0 + lane] : j0 + lane) : 0;
        if (lane < nb) {
            J = jobs[jid];
            D = descs[jid];
            ok = dec_job_ok(J, D, STYLED) && J.cw <= 8 * Q;
            if (!ok) atomicCAS(err, 0u, (uint32_t)J2K_DEVERR_BAD_JOB);
        }
        const unsigned okmask = __ballot_sync(~0u, ok);
        for (int i = lane; i < S.kCols * L; i += 32) S.w[i] = 0;
        if (Q < 8)  // (only the bytes of words that there are get written below)
            for (int i = lane; i < 2 * L; i += 32) S.colset(i & 1, i >> 1) = 0;
        for (int b = 0; b < nb; ++b) {
            if (!((okmask >> b) & 1)) continue;
            const int cw = __shfl_sync(~0u, (int)J.cw, b), ch = __shfl_sync(~0u, (int)J.ch, b);
            const size_t pitch = __shfl_sync(~0u, J.pitch, b);
            int32_t* blk = coeff + __shfl_sync(~0u, (unsigned long long)J.off, b);
            for (int r = lane / WX; r < ch; r += WY)
                for (int x = lane % WX; x < cw; x += WX) blk[(size_t)r * pitch + x] = 0;
        }
        // this lane's block, and the sizes and pass counts of the blocks of its items
        const int np = ok && D.numbps > 0 ? min((int)D.npasses, 3 * (int)D.numbps - 2) : 0;
        StripeLane<L, Q> me{S,    LaneMem<L, Q>(S, tabs, J.orient & 3, lane < L ? lane : 0),
                            lane, J.cw, J.ch, {}, {}, false};
        int icw[R], ich[R], inp[R], inb[R];
        uint32_t ipitch[R];
        int32_t* iblk[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int i = lane + 32 * r, b = (i / Q) & 31;
            icw[r] = __shfl_sync(~0u, (int)J.cw, b);
            ich[r] = __shfl_sync(~0u, (int)J.ch, b);
            inp[r] = __shfl_sync(~0u, np, b);
            inb[r] = __shfl_sync(~0u, (int)D.numbps, b);
            ipitch[r] = __shfl_sync(~0u, J.pitch, b);
            iblk[r] = coeff + __shfl_sync(~0u, (unsigned long long)J.off, b);
            if (i >= Q * L) inp[r] = 0;
        }
        // With one word a stripe and up to 4 blocks a lane per column prepares it (with 8, two columns a
        // lane, that is no faster): the columns of block lane / 8
        constexpr bool COLS = Q == 1 && L <= 4;
        int xcw = 0, xch = 0, xnp = 0, xnb = 0;
        if constexpr (COLS) {
            xcw = __shfl_sync(~0u, (int)J.cw, lane >> 3);
            xch = __shfl_sync(~0u, (int)J.ch, lane >> 3);
            xnp = __shfl_sync(~0u, np, lane >> 3);
            xnb = __shfl_sync(~0u, (int)D.numbps, lane >> 3);
            if (lane >= 8 * L) xnp = 0;
        }
        const int pmax = __reduce_max_sync(~0u, np > 0 ? (int)D.numbps : 0);
        const int smax = (__reduce_max_sync(~0u, np > 0 ? (int)J.ch : 0) + 3) >> 2;
        const int st = STYLED ? (job_style ? (int)job_style[jid] : style) : 0;
        __syncwarp();
        // t = 3 * bit-plane + 2, 1, 0 for its three passes: the blocks of a warp code the same
        // plane at the same time (their lowest planes, which hold most symbols, are alike; counted
        // from the first pass they would be apart by the difference of their plane counts)
        for (int t = 3 * pmax - 1; t >= 0; --t) {
            const int p = t / 3, kind = kPassCU - t % 3;
            auto pass_of = [&](int numbps) { return 3 * (numbps - 1 - p) - t % 3; };  // its number in the block
            const int q = pass_of(D.numbps);
            const bool on = q >= 0 && q < np;
            if (on)
                me.template begin<STYLED>(q, D.npasses, bytes + D.offset, D.length, st,
                                          STYLED ? pass_ends + (size_t)jid * J2K_PASS_STRIDE : nullptr);
            bool ion[R];
#pragma unroll
            for (int r = 0; r < R; ++r) ion[r] = pass_of(inb[r]) >= 0 && pass_of(inb[r]) < inp[r];
            const bool xon = pass_of(xnb) >= 0 && pass_of(xnb) < xnp;
            for (int s = 0; s < smax; ++s) {
                if (COLS && kind != kPassMR) {
                    const int b = lane >> 3, x = lane & 7;
                    const bool mine = xon && 4 * s < xch;
                    bool has = false;
                    if constexpr (COLS)
                        has = mine && x < xcw && stripe_prepare_column(S, kind, s, x, b, stripe_rows(xch, s));
                    const unsigned set = __ballot_sync(~0u, has);
                    if (mine && x == 0) {
                        S.cols(b)[0] = (uint8_t)(set >> (lane & 24));
                        if (kind == kPassSP) S.vis(s, 0, b) = 0;  // (a stripe without symbols is not finished)
                    }
                }
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const int i = lane + 32 * r;
                    if (ion[r] && 4 * s < ich[r] && (!COLS || kind == kPassMR)) {
                        if (kind == kPassMR) stripe_prepare_mr(S, s, i % Q, i / Q, icw[r]);
                        else stripe_prepare_zc(S, kind, s, i % Q, i / Q, icw[r], stripe_rows(ich[r], s));
                    }
                }
                __syncwarp();
                // (with one word a stripe, preparing and finishing it costs as much as its symbols)
                if (Q == 1 && !__any_sync(~0u, on && 4 * s < me.ch && S.colset(0, lane) != 0)) {
                    __syncwarp();
                    continue;
                }
                if (on && 4 * s < me.ch) {
                    const uint32_t rv = stripe_rows(me.ch, s);
                    if (kind == kPassSP) me.template decode_zc<STYLED, kPassSP>(rv);
                    else if (kind == kPassMR) me.template decode_mr<STYLED>();
                    else me.template decode_zc<STYLED, kPassCU>(rv);
                }
                __syncwarp();
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const int i = lane + 32 * r;
                    if (ion[r] && 4 * s < ich[r]) {
                        const uint32_t ones = kind == kPassMR
                                                  ? stripe_finish_mr(S, s, i % Q, i / Q, icw[r])
                                                  : stripe_finish_zc(S, kind, s, i % Q, i / Q, icw[r]);
                        stripe_add_bits(ones, iblk[r], ipitch[r], s, i % Q, p);
                    }
                }
                __syncwarp();
            }
        }
        // signs, and the middle of the undecoded interval of a cut block
        const int32_t my_half = ok ? cut_half(D.numbps, D.npasses) : 0;
        for (int b = 0; b < nb; ++b) {
            if (!((okmask >> b) & 1)) continue;
            const int cw = __shfl_sync(~0u, (int)J.cw, b), ch = __shfl_sync(~0u, (int)J.ch, b);
            const size_t pitch = __shfl_sync(~0u, J.pitch, b);
            int32_t* blk = coeff + __shfl_sync(~0u, (unsigned long long)J.off, b);
            const int32_t half = __shfl_sync(~0u, my_half, b);
            for (int r = lane / WX; r < ch; r += WY)
                for (int x = lane % WX; x < cw; x += WX) {
                    const int sh = 4 * (x & 7) + (r & 3);
                    int32_t v = __ldcg(blk + (size_t)r * pitch + x);
                    if ((S.sig(r >> 2, x >> 3, b) >> sh) & 1) v += half;
                    if ((S.neg(r >> 2, x >> 3, b) >> sh) & 1) v = -v;
                    blk[(size_t)r * pitch + x] = v;
                }
        }
        __syncwarp();
        int nx = 0;
        if (lane == 0) nx = (int)(gridDim.x * (blockDim.x >> 5) + atomicAdd(queue, 1u));
        g = __shfl_sync(~0u, nx, 0);
    }
}

constexpr size_t kTablesBytes = (sizeof(DecTables) + 15) & ~(size_t)15;
// warps per CTA of the one-symbol-per-step decoder for L blocks per warp: 32 blocks per CTA for
// L >= 8, four warps for smaller L (so that a CTA's shared-memory state stays near 70 KB or less)
template <int L>
__host__ __device__ constexpr int cta_warps() {
    return L >= 8 ? 32 / L : 4;
}

template <int L>
__host__ __device__ constexpr size_t lanes_smem_bytes() {
    return kTablesBytes + (size_t)cta_warps<L>() * lane_state_bytes<L>();
}

// symbol kinds and pending symbols of decode_block_steps
enum : int { kSymZC = 0, kSymSign = 1, kSymMR = 2, kSymRL = 3, kSymUni = 4 };
enum : int { kPendNone = 0, kPendSign = 1, kPendUni1 = 2, kPendUni2 = 3 };

// The same decode as decode_block (unstyled blocks), written as a loop of one symbol per step:
// (1) advance the cursor (pass, stripe, column, row) to the next sample that codes a symbol in its
// pass, or take the pending sign / run-length index symbol, (2) decode that one symbol -- the MQ
// decoder's only call site -- and (3) apply it.  Lanes of a warp that decode different blocks
// with it stay together on the decoding step whatever pass or column each is in.  The scan
// order, contexts and pass rules are T.800 D.3-D.5 (significance propagation, magnitude
// refinement and cleanup passes, stripes of four rows scanned column by column, the cleanup
// pass's run-length mode).  Host-callable, for the tests.
template <bool RED = false, class State>
__host__ __device__ void decode_block_steps(State& S, const DecTables& tabs, const uint8_t* data, int len, int numbps,
                                            int npasses, int orient, int cw, int ch, int32_t* blk, size_t pitch,
                                            bool active = true) {
    auto add_bit = [&](int x, int y, int p) {
#ifdef __CUDA_ARCH__
        if (RED) {
            atomicOr(reinterpret_cast<unsigned int*>(blk + (size_t)y * pitch + x), 1u << p);
            return;
        }
#endif
        blk[(size_t)y * pitch + x] |= 1 << p;
    };
    const uint8_t* zct = tabs.zc[orient & 3];
    const uint32_t* mq = tabs.mq;
    const int np = npasses;
    const uint64_t cols = cw >= 64 ? ~0ull : ((1ull << cw) - 1);
    Mqd m;
    if (active) {
        for (int c = 0; c < 19; ++c) S.st(c) = 0;
        S.st(0) = 4 << 1;
        S.st(17) = 3 << 1;
        S.st(18) = 46 << 1;
        m.init(data, len);
    }
    // cursor
    int pass = 0, ptype = kPassCU, p = numbps - 1, y0 = 0, x = 0, k = 4, ny = min(4, ch);
    int pending = kPendNone, idx = 0;
    bool colstart = false, nwv = false;
    uint32_t W = 0, NW = 0, V = 0, R = 0;
    uint64_t cm = 0;
    // candidate columns of the stripe at y0 in the current pass
    auto stripe_setup = [&]() {
        ny = min(4, ch - y0);
        uint64_t c = 0;
        for (int r = 0; r < ny; ++r) {
            const uint64_t own = S.sig(y0 + r + 1);
            if (ptype == kPassSP) {
                uint64_t nbm = S.sig(y0 + r) | own | S.sig(y0 + r + 2);
                nbm |= (nbm << 1) | (nbm >> 1);
                c |= ~own & nbm;
            } else {
                const uint64_t vis = S.vis(y0 + r + 1);
                c |= (ptype == kPassMR ? own : ~own) & ~vis;
            }
        }
        cm = c & cols;
    };
    auto colw = [&](bool negs) -> uint32_t {
        uint32_t w = 0;
        for (int r = 0; r < 6; ++r) w |= nb3(negs ? S.neg(y0 + r) : S.sig(y0 + r), x) << (3 * r);
        return w;
    };
    if (active) stripe_setup();
    // rows of the current column, from row k on, that code a symbol in this pass
    auto cand_rows = [&]() -> uint32_t {
        const uint32_t s4 = ((W >> 4) & 1) | ((W >> 6) & 2) | ((W >> 8) & 4) | ((W >> 10) & 8);
        uint32_t rows;
        if (ptype == kPassSP) {
            uint32_t n4 = 0;
            for (int r = 0; r < 4; ++r) n4 |= (uint32_t)(((W >> (3 * r)) & 0x1EF) != 0) << r;
            rows = ~s4 & n4;
        } else {
            rows = (ptype == kPassMR ? s4 : ~s4) & ~V;
        }
        return rows & ((1u << ny) - 1) & (0xFu << k);
    };
    // On the device every lane of the warp runs this loop (lanes without a block, or done with
    // theirs, inactive), and the vote at the top of each step brings the lanes back together
    // before the next symbol, however their searches diverged.
#ifdef __CUDA_ARCH__
    while (__any_sync(0xffffffffu, active)) {
        if (!active) continue;
#else
    while (active) {
#endif
        int kind = kSymUni;
        if (pending == kPendSign) {
            kind = kSymSign;
        } else if (pending == kPendNone) {
            bool done = false;
            for (;;) {
                if (k < 4) {
                    if (ptype == kPassCU && colstart && ny == 4 && W == 0 && V == 0) {
                        kind = kSymRL;  // run-length mode: no significant sample around the column
                        break;
                    }
                    const uint32_t rows = cand_rows();
                    if (rows) {
                        k = ctz64(rows);
                        kind = ptype == kPassMR ? kSymMR : kSymZC;
                        break;
                    }
                    k = 4;
                }
                if (cm) {  // next column of the stripe that holds a candidate
                    x = ctz64(cm);
                    cm &= cm - 1;
                    W = colw(false);
                    nwv = false;
                    V = 0;
                    R = 0;
                    if (ptype != kPassSP)
                        for (int r = 0; r < ny; ++r) V |= (uint32_t)((S.vis(y0 + r + 1) >> x) & 1) << r;
                    if (ptype == kPassMR)
                        for (int r = 0; r < ny; ++r) R |= (uint32_t)((S.ref(y0 + r + 1) >> x) & 1) << r;
                    k = 0;
                    colstart = true;
                    continue;
                }
                if (y0 + 4 < ch) {  // next stripe
                    y0 += 4;
                    stripe_setup();
                    continue;
                }
                // end of the pass
                if (ptype == kPassCU)
                    for (int r = 0; r < 66; ++r) S.vis(r) = 0;
                if (++pass >= np || (ptype == kPassCU && p == 0)) {  // (the last plane's cleanup ends it)
                    done = true;
                    break;
                }
                if (ptype == kPassCU) {
                    --p;
                    ptype = kPassSP;
                } else {
                    ptype = ptype == kPassSP ? kPassMR : kPassCU;
                }
                y0 = 0;
                stripe_setup();
            }
            if (done) {
                active = false;
                continue;
            }
        }
        // the symbol's context (sign symbols: label | xor bit << 7)
        int cx, xr = 0;
        if (kind == kSymZC) {
            cx = zct[(W >> (3 * k)) & 511];
        } else if (kind == kSymMR) {
            cx = ((R >> k) & 1) ? 16 : (((W >> (3 * k)) & 0x1EF) ? 15 : 14);
        } else if (kind == kSymSign) {
            if (!nwv && W) {  // (with no significant neighbour the signs around do not matter)
                NW = colw(true);
                nwv = true;
            }
            const int sc = tabs.sc[sign_nbhd(W, NW, k)];
            cx = sc & 31;
            xr = sc >> 7;
        } else {
            cx = kind == kSymRL ? 17 : 18;
        }
        const int d = m.decode(S.st(cx), mq) ^ xr;
        if (kind == kSymZC) {
            if (ptype == kPassSP) S.vis(y0 + k + 1) |= 1ull << x;
            if (d) pending = kPendSign;
            else ++k;
            colstart = false;
        } else if (kind == kSymSign) {
            const int y = y0 + k;
            S.sig(y + 1) |= 1ull << x;
            if (d) S.neg(y + 1) |= 1ull << x;
            add_bit(x, y, p);
            W |= 1u << (3 * k + 4);
            NW |= (uint32_t)d << (3 * k + 4);
            if (ptype == kPassSP) cm |= (2ull << x) & cols;
            pending = kPendNone;
            ++k;
        } else if (kind == kSymMR) {
            const int y = y0 + k;
            if (d) add_bit(x, y, p);
            S.ref(y + 1) |= 1ull << x;
            ++k;
        } else if (kind == kSymRL) {
            colstart = false;
            if (d) pending = kPendUni1;
            else k = 4;
        } else if (pending == kPendUni1) {
            idx = d << 1;
            pending = kPendUni2;
        } else {
            k = idx | d;
            pending = kPendSign;
        }
    }
}

// One code-block per lane, each decoded by decode_block_steps.

template <int L>
__global__ void __launch_bounds__(32 * cta_warps<L>())
t1_decode_steps_kernel(const j2k_cb_desc* __restrict__ descs, const uint8_t* __restrict__ bytes,
                       const j2k_cb_job* __restrict__ jobs, int njobs, int32_t* __restrict__ coeff,
                       uint32_t* __restrict__ err) {
    extern __shared__ __align__(16) uint8_t dsm[];
    DecTables& tabs = *reinterpret_cast<DecTables*>(dsm);
    for (int i = threadIdx.x; i < 4 * 512; i += blockDim.x) fill_tables_entry(tabs, i);
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int j0 = (blockIdx.x * cta_warps<L>() + wid) * L;
    if (j0 >= njobs) return;
    const int nb = min(L, njobs - j0);
    uint8_t* wsm = dsm + kTablesBytes + (size_t)wid * lane_state_bytes<L>();
    uint64_t* base = reinterpret_cast<uint64_t*>(wsm);
    uint8_t* stb = wsm + (size_t)4 * 66 * L * 8;
    j2k_cb_job J{};
    j2k_cb_desc D{};
    bool ok = false;
    if (lane < nb) {
        J = jobs[j0 + lane];
        D = descs[j0 + lane];
        ok = dec_job_ok(J, D, false);
        if (!ok) atomicCAS(err, 0u, (uint32_t)J2K_DEVERR_BAD_JOB);
    }
    const unsigned okmask = __ballot_sync(~0u, ok);
    for (int i = lane; i < 4 * 66 * L; i += 32) base[i] = 0;
    for (int b = 0; b < nb; ++b) {
        if (!((okmask >> b) & 1)) continue;
        const int cw = __shfl_sync(~0u, (int)J.cw, b), ch = __shfl_sync(~0u, (int)J.ch, b);
        const size_t pitch = __shfl_sync(~0u, J.pitch, b);
        int32_t* blk = coeff + __shfl_sync(~0u, (unsigned long long)J.off, b);
        for (int r = 0; r < ch; ++r)
            for (int x = lane; x < cw; x += 32) blk[(size_t)r * pitch + x] = 0;
    }
    __syncwarp();
    {  // every lane of the warp takes part in the step loop, whether or not it has a block
        LaneState<L> S{base, stb, lane < L ? lane : 0};
        const bool act = ok && D.numbps > 0 && D.npasses > 0;
        decode_block_steps<true>(S, tabs, bytes + D.offset, D.length, D.numbps, D.npasses, J.orient, J.cw, J.ch,
                                 coeff + J.off, J.pitch, act);
    }
    __syncwarp();
    const int32_t my_half = ok ? cut_half(D.numbps, D.npasses) : 0;
    for (int b = 0; b < nb; ++b) {
        if (!((okmask >> b) & 1)) continue;
        const int cw = __shfl_sync(~0u, (int)J.cw, b), ch = __shfl_sync(~0u, (int)J.ch, b);
        const size_t pitch = __shfl_sync(~0u, J.pitch, b);
        int32_t* blk = coeff + __shfl_sync(~0u, (unsigned long long)J.off, b);
        const int32_t half = __shfl_sync(~0u, my_half, b);
        for (int r = 0; r < ch; ++r) {
            const uint64_t sg = base[(0 * 66 + r + 1) * L + b], ng = base[(1 * 66 + r + 1) * L + b];
            for (int x = lane; x < cw; x += 32) {
                int32_t v = __ldcg(blk + (size_t)r * pitch + x);
                if ((sg >> x) & 1) v += half;
                if ((ng >> x) & 1) v = -v;
                blk[(size_t)r * pitch + x] = v;
            }
        }
    }
}

}  // namespace

// Host execution of the device decoder logic for one block (used by the test suite): the stripe
// decoder that the default kernel runs, its warp-wide parts one item after another, or (steps) the
// one-symbol-per-step loop of J2K_TUNE_T1D_STEPS.
template <bool STYLED, int Q>
static void decode_stripes_host(const uint8_t* data, int len, int numbps, int npasses, int orient, int cw, int ch,
                                int32_t* out, size_t pitch, int style, const uint32_t* pe) {
    static const StripeTables T = [] {  // built once, thread-safely
        StripeTables t{};
        for (int i = 0; i < 4 * 512; ++i) fill_stripe_tables_entry(t, i);
        return t;
    }();
    uint32_t words[stripe_state_words<1, Q>()] = {};
    const StripeState<1, Q> S{words};
    StripeLane<1, Q> me{S, LaneMem<1, Q>(S, T, orient, 0), 0, cw, ch, {}, {}, false};
    const int np = std::min(npasses, 3 * numbps - 2), ns = (ch + 3) / 4;
    for (int q = 0; q < np; ++q) {
        const int kind = q == 0 ? kPassCU : (q + 2) % 3, p = numbps - 1 - (q + 2) / 3;
        me.template begin<STYLED>(q, npasses, data, len, style, pe);
        for (int s = 0; s < ns; ++s) {
            const uint32_t rv = stripe_rows(ch, s);
            for (int i = 0; i < Q; ++i) {
                if (kind == kPassMR) stripe_prepare_mr(S, s, i, 0, cw);
                else stripe_prepare_zc(S, kind, s, i, 0, cw, rv);
            }
            if (kind == kPassSP) me.template decode_zc<STYLED, kPassSP>(rv);
            else if (kind == kPassMR) me.template decode_mr<STYLED>();
            else me.template decode_zc<STYLED, kPassCU>(rv);
            for (int i = 0; i < Q; ++i) {
                const uint32_t ones = kind == kPassMR ? stripe_finish_mr(S, s, i, 0, cw)
                                                      : stripe_finish_zc(S, kind, s, i, 0, cw);
                stripe_add_bits(ones, out, pitch, s, i, p);
            }
        }
    }
    for (int y = 0; y < ch; ++y)
        for (int x = 0; x < cw; ++x)
            if ((S.neg(y >> 2, x >> 3, 0) >> (4 * (x & 7) + (y & 3))) & 1)
                out[(size_t)y * pitch + x] = -out[(size_t)y * pitch + x];
}

static int decode_block_host(const uint8_t* data, int len, int numbps, int npasses, int orient, int cw, int ch,
                             int32_t* out, size_t pitch, bool steps) {
    if (cw < 1 || ch < 1 || cw > 64 || ch > 64 || orient < 0 || orient > 3 || numbps < 0 || numbps > 31 ||
        npasses < 0 || npasses > 3 * numbps || len < 0 || (len > 0 && !data) || !out || pitch < (size_t)cw)
        return -1;  // the checks the kernel makes of a descriptor, and the host buffers
    for (int y = 0; y < ch; ++y)
        for (int x = 0; x < cw; ++x) out[(size_t)y * pitch + x] = 0;
    if (numbps == 0 || npasses == 0) return 0;
    if (!steps) {
        const auto decode = cw <= 8 ? decode_stripes_host<false, 1> : decode_stripes_host<false, 8>;
        decode(data, len, numbps, npasses, orient, cw, ch, out, pitch, 0, nullptr);
        return 0;
    }
    DecSmem S;
    for (int r = 0; r < 66; ++r) S.sig_[r] = S.neg_[r] = S.ref_[r] = S.vis_[r] = 0;
    for (int k = 0; k < 19; ++k) S.st_[k] = 0;
    static const DecTables T = [] {  // built once, thread-safely
        DecTables t{};
        for (int i = 0; i < 4 * 512; ++i) fill_tables_entry(t, i);
        return t;
    }();
    decode_block_steps(S, T, data, len, numbps, npasses, orient, cw, ch, out, pitch);
    for (int y = 0; y < ch; ++y)
        for (int x = 0; x < cw; ++x)
            if ((S.neg_[y + 1] >> x) & 1) out[(size_t)y * pitch + x] = -out[(size_t)y * pitch + x];
    return 0;
}

extern "C" int j2k_t1_decode_block_host(const uint8_t* data, int len, int numbps, int npasses, int orient,
                                        int cw, int ch, int32_t* out, size_t pitch) {
    return decode_block_host(data, len, numbps, npasses, orient, cw, ch, out, pitch, false);
}

extern "C" int j2k_t1_decode_block_steps_host(const uint8_t* data, int len, int numbps, int npasses, int orient,
                                              int cw, int ch, int32_t* out, size_t pitch) {
    return decode_block_host(data, len, numbps, npasses, orient, cw, ch, out, pitch, true);
}

// The same for a block coded with a code-block style, its segments located by pass_ends
// (J2K_PASS_STRIDE entries; values past len are clamped to it, as the kernel does).
extern "C" int j2k_t1_decode_block_styled_host(const uint8_t* data, int len, const uint32_t* pass_ends, int numbps,
                                               int npasses, int orient, int style, int cw, int ch, int32_t* out,
                                               size_t pitch) {
    if (cw < 1 || ch < 1 || cw > 64 || ch > 64 || orient < 0 || orient > 3 || numbps < 0 || numbps > 31 ||
        npasses < 0 || npasses > 3 * numbps || npasses > J2K_PASS_STRIDE - 1 || len < 0 || (len > 0 && !data) ||
        !out || pitch < (size_t)cw || !pass_ends || style < 0 || style > 7)
        return -1;
    for (int y = 0; y < ch; ++y)
        for (int x = 0; x < cw; ++x) out[(size_t)y * pitch + x] = 0;
    const auto decode = cw <= 8 ? decode_stripes_host<true, 1> : decode_stripes_host<true, 8>;
    if (numbps > 0 && npasses > 0)
        decode(data, len, numbps, npasses, orient, cw, ch, out, pitch, style, pass_ends);
    return 0;
}

template <bool STYLED, int L, int Q>
static j2k_status launch_stripe(j2k_ctx* ctx, cudaStream_t st, const j2k_cb_desc* descs, const uint8_t* bytes,
                                const j2k_cb_job* d_jobs, size_t njobs, int32_t* coeff, int style,
                                const uint32_t* pass_ends, const uint8_t* job_style, const uint32_t* order,
                                const uint32_t* keys) {
    static std::atomic<uint64_t> attr_set{0};  // devices whose attribute is set, per instantiation
    const uint64_t bit = 1ull << (ctx->device & 63);
    if (!(attr_set.load() & bit)) {
        J2K_CUDA(ctx, cudaFuncSetAttribute(t1_decode_stripe_kernel<STYLED, L, Q>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)stripe_smem_bytes<L, Q>(stripe_warps<L, Q>())));
        attr_set.fetch_or(bit);
    }
    uint32_t* queue = (uint32_t*)j2k_scratch(ctx, SCR_DECQ, 4);
    if (!queue) return J2K_ERR_OUT_OF_MEMORY;
    J2K_CUDA(ctx, cudaMemsetAsync(queue, 0, 4, st));
    // the groups spread over the SMs first, then over the warps of a CTA
    const size_t sms = (size_t)ctx->sm_count, resident = sms * stripe_warps<L, Q>();
    // blocks that can have a warp alone with all blocks still resident at once
    const size_t alone = L > 1 && keys && resident * L > njobs ? std::min(njobs, (resident * L - njobs) / (L - 1)) : 0;
    const size_t groups = alone + (njobs - alone + L - 1) / L;
    const unsigned grid = (unsigned)std::min(groups, sms);
    const int warps = (int)std::min<size_t>((groups + grid - 1) / grid, (size_t)stripe_warps<L, Q>());
    t1_decode_stripe_kernel<STYLED, L, Q><<<grid, 32 * warps, stripe_smem_bytes<L, Q>(warps), st>>>(
        descs, bytes, d_jobs, (int)njobs, coeff, ctx->d_err, style, pass_ends, job_style, order, keys, (int)alone, queue);
    J2K_CUDA(ctx, cudaGetLastError());
    return J2K_OK;
}

// keys[i] = codeword length of job i, ids[i] = i
__global__ void t1d_order_keys(const j2k_cb_desc* __restrict__ descs, int n, uint32_t* __restrict__ keys,
                               uint32_t* __restrict__ ids) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int32_t len = descs[i].length;
    keys[i] = len > 0 ? (uint32_t)len : 0u;
    ids[i] = (uint32_t)i;
}

// The jobs sorted by codeword length, longest first (a stable radix sort: equal lengths keep
// their list order), in scratch; nullptr with the error set when scratch runs out.
// *keys: the lengths in that order.
static const uint32_t* decode_order(j2k_ctx* ctx, cudaStream_t st, const j2k_cb_desc* descs, size_t njobs,
                                    const uint32_t** keys) {
    const int n = (int)njobs;
    size_t tmp = 0;
    cub::DeviceRadixSort::SortPairsDescending(nullptr, tmp, (const uint32_t*)nullptr, (uint32_t*)nullptr,
                                              (const uint32_t*)nullptr, (uint32_t*)nullptr, n, 0, 32, st);
    const size_t words = 4 * njobs + 64;
    uint32_t* w = (uint32_t*)j2k_scratch(ctx, SCR_DECORD, words * 4 + tmp + 64);
    if (!w) return nullptr;
    uint32_t *keys_in = w, *keys_out = w + njobs, *ids_in = w + 2 * njobs, *ids_out = w + 3 * njobs;
    void* temp = w + words;
    t1d_order_keys<<<(unsigned)((njobs + 255) / 256), 256, 0, st>>>(descs, n, keys_in, ids_in);
    if (j2k_cuda_check(ctx, cudaGetLastError(), "decode order keys") != J2K_OK) return nullptr;
    if (j2k_cuda_check(ctx, cub::DeviceRadixSort::SortPairsDescending(temp, tmp, keys_in, keys_out, ids_in, ids_out,
                                                                      n, 0, 32, st),
                       "decode order sort") != J2K_OK)
        return nullptr;
    *keys = keys_out;
    return ids_out;
}

template <int L>
static j2k_status launch_steps(j2k_ctx* ctx, cudaStream_t st, const j2k_cb_desc* descs,
                               const uint8_t* bytes, const j2k_cb_job* d_jobs, size_t njobs, int32_t* coeff) {
    constexpr size_t smem = lanes_smem_bytes<L>();
    const unsigned grid = (unsigned)((njobs + L * cta_warps<L>() - 1) / (L * cta_warps<L>()));
    static std::atomic<uint64_t> attr_set{0};
    const uint64_t bit = 1ull << (ctx->device & 63);
    if (!(attr_set.load() & bit)) {
        J2K_CUDA(ctx, cudaFuncSetAttribute(t1_decode_steps_kernel<L>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)smem));
        attr_set.fetch_or(bit);
    }
    t1_decode_steps_kernel<L><<<grid, 32 * cta_warps<L>(), smem, st>>>(descs, bytes, d_jobs, (int)njobs, coeff,
                                                                            ctx->d_err);
    J2K_CUDA(ctx, cudaGetLastError());
    return J2K_OK;
}

// Blocks per warp by the work there is, as a number of blocks of the largest one's size: one while
// those would be resident at once that way (16 an SM), two up to 40 an SM, four for more (the long
// blocks get warps of their own as far as all still fit).  A block runs fastest alone; sharing a warp
// saves instructions, which counts once the ALU pipes are full, and that is a matter of how many
// blocks wait behind one another, not of how large they are.  Host to host on B200, 1 / 2 / 4 / 8
// blocks per warp: 70 blocks of a 512 x 512 gray image 5.5 ms, with two 7.6, four 10.2; 777 of
// 1024 x 1024 colour 6.7, 8.4, 10.4; 24 images of mixed sizes and block sizes (the work of 1590 largest
// blocks) 11.0 / 11.2 / 13.6 / 17.5; 3072 blocks of 2048 x 2048 colour 12.4 / 10.0 / 11.1 / 13.9; 12288
// blocks of 4096 x 4096 colour 42 / 32 / 20.0 / 21.6.  Smaller blocks, 1 / 2 / 4 / 8: 3072 of 32 x 32
// (1024 x 1024 colour) 4.0 / 3.5 / 3.8 / 4.7; 12288 of 32 x 32 (2048 x 2048) 14.9 / 11.8 / 8.5 / 9.7; 4096
// of 16 x 16 (1024 x 1024 gray) 1.45 / 1.24 / 1.36 / 1.57; 12288 of 16 x 16 4.1 / 3.2 / 2.2 / 2.5.
// Blocks up to 8 wide are one word a stripe, with little state, few symbols at a time and the more so
// as they are many: up to 16 a warp.  Host to host, 1 / 2 / 4 / 8 / 16: 4096 of 8 x 32 (1024 x 1024 gray)
// 1.59 / 1.41 / 1.43 / 1.56 / 1.71; 6168 of 8 x 64 (1024 x 1024 colour) 4.0 / 3.3 / 3.6 / 3.6 / 4.1; 12336
// of 4 x 64 4.3 / 3.2 / 2.6 / 2.6 / 2.8; 24576 of 8 x 64 (2048 x 2048 colour) 16.6 / 13.0 / 9.4 / 7.1 / 7.3;
// 49152 of 8 x 32 16.5 / 13.0 / 10.2 / 7.4 / 6.4; 196608 of 8 x 8 16.5 / 12.2 / 9.6 / 7.5 / 6.1.
// In a mixed set a block counts as a quarter of the largest one at least, so that one image with large
// blocks does not hide thousands of small ones: the codestreams of 30 images of 512 x 512 gray with
// 16 x 16 blocks and one of 64 x 64 with 64 x 64 take 12.6 ms with one block per warp, 9.0 with four.
static int stripe_blocks_per_warp(const j2k_ctx* ctx, size_t njobs, size_t samples, int cbw, int cbh) {
    const size_t n = std::max(samples / ((size_t)cbw * cbh), njobs / 4), sms = (size_t)ctx->sm_count;
    if (cbw > 8) return n <= 16 * sms ? 1 : (n <= 40 * sms ? 2 : 4);
    return n <= 16 * sms ? 1 : (n <= 48 * sms ? 2 : (n <= 96 * sms ? 4 : (n <= 256 * sms ? 8 : 16)));
}

template <bool STYLED, int Q, class... Args>
static j2k_status launch_stripe_lanes(int lanes, Args... args) {
    switch (lanes) {
    case 1: return launch_stripe<STYLED, 1, Q>(args...);
    case 2: return launch_stripe<STYLED, 2, Q>(args...);
    case 4: return launch_stripe<STYLED, 4, Q>(args...);
    case 8: return launch_stripe<STYLED, 8, Q>(args...);
    default: return launch_stripe<STYLED, 16, Q>(args...);
    }
}

j2k_status j2k_t1_decode_jobs(j2k_ctx* ctx, const j2k_cb_desc* descs, const uint8_t* bytes,
                              const j2k_cb_job* d_jobs, size_t njobs, size_t samples, int cbw, int cbh, int32_t* coeff,
                              cudaStream_t st, int style, const uint32_t* pass_ends, const uint8_t* job_style) {
    if (njobs == 0) return J2K_OK;
    if ((style || job_style) && !pass_ends)
        return j2k_fail(ctx, J2K_ERR_INVALID_ARG, "a styled decode needs the pass ends");
    const bool styled = style || job_style;
    const int forced = ctx->t1d_lanes;
    if (!styled && ctx->t1d_steps) {
        switch (forced) {
        case 8: return launch_steps<8>(ctx, st, descs, bytes, d_jobs, njobs, coeff);
        case 16: return launch_steps<16>(ctx, st, descs, bytes, d_jobs, njobs, coeff);
        case 32: return launch_steps<32>(ctx, st, descs, bytes, d_jobs, njobs, coeff);
        default: break;
        }
    }
    const int L = forced < 0 ? stripe_blocks_per_warp(ctx, njobs, samples, cbw, cbh)
                             : (forced <= 1 ? 1 : (forced == 2 ? 2 : (forced <= 4 ? 4 : (forced <= 8 ? 8 : 16))));
    const uint32_t *ord = nullptr, *keys = nullptr;
    if (ctx->t1d_order && njobs > (size_t)L) {
        ord = decode_order(ctx, st, descs, njobs, &keys);
        if (!ord) return J2K_ERR_OUT_OF_MEMORY;
    }
    const auto go = [&](auto... a) {
        return styled ? (cbw <= 8 ? launch_stripe_lanes<true, 1>(L, a...) : launch_stripe_lanes<true, 8>(L, a...))
                      : (cbw <= 8 ? launch_stripe_lanes<false, 1>(L, a...) : launch_stripe_lanes<false, 8>(L, a...));
    };
    return go(ctx, st, descs, bytes, d_jobs, njobs, coeff, style, pass_ends, job_style, ord, keys);
}
