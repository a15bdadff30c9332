// EBCOT tier-1 encoder: context modelling (a warp per code-block) + MQ coding (a warp pair for 1 to 32
// code-blocks).
//
// Reference: src/CL/oclbpc.cl:279-746 via src/OCLBPC.cpp:38-50.  The reference kernel computes
// the MSB plane and sigma/neighbourhood state only (its coding actions are empty comments,
// oclbpc.cl:388-443,625-740); the passes, scan order and state variables it documents
// (oclbpc.cl:19-111) are completed here from ITU-T T.800 Annex D (contexts, run-length mode,
// sign coding) and Annex C (MQ coder).
//
// Phase A — one warp per code-block writes the exact (context, decision) sequence of the serial
// coder (t1sym.cuh), one byte per symbol: label in bits 0-4, decision in bit 7; sign symbols also
// carry their context's XOR bit in bit 5, so that a raw-coded pass can recover the sign itself.
//
// Phase B — the MQ encoder over the symbol streams (T.800 C.2, FLUSH of C.2.9, trailing 0xFF dropped;
// mq_enc.cuh), a block on one lane of each of two warps: the interval chain and the byte output.
// Codeword bytes are written as aligned 32-bit words.
#include <cub/cub.cuh>

#include <algorithm>

#include "j2k_internal.cuh"

namespace {

constexpr int kWarpsPerCta = 8;
constexpr int kRows = 64;
constexpr int kPlaneWords = 32 * kRows;  // per-block bit-plane scratch: 64 rows x 32 planes

// warp exclusive prefix sum; returns the total in *tot
__device__ __forceinline__ int warp_excl(int v, int lane, int* tot) {
    int inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    *tot = __shfl_sync(0xffffffffu, inc, 31);
    return inc - v;
}

#include "t1sym.cuh"

// MINB: resident CTAs per SM the register budget is cut for (2: 128 registers, no spills; 3: 80, with
// 220 bytes of spill stores and 504 of loads in all forms together, and more warps to hide the ALU
// chains: 256 images of mixed sizes take 3.70 ms with either)
template <int MINB>
__global__ void __launch_bounds__(kWarpsPerCta * 32, MINB)
t1_symbols_kernel(const int32_t* __restrict__ coeff, const j2k_cb_job* __restrict__ jobs,
                  int njobs, const uint32_t* __restrict__ order, uint32_t* __restrict__ queue,
                  uint8_t* __restrict__ syms, uint32_t* __restrict__ nsyms,
                  uint32_t* __restrict__ pass_end, uint64_t* __restrict__ plane_scratch,
                  j2k_cb_desc* __restrict__ descs, uint32_t* __restrict__ err, int pad) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    extern __shared__ __align__(16) uint8_t sym_smem[];
    SymSmem& S = reinterpret_cast<SymSmem*>(sym_smem)[wid];
    // persistent: each warp pulls code-blocks from the device-side queue until it is empty;
    // its bit-plane scratch slot is reused from block to block
    uint64_t* planes = plane_scratch + (size_t)(blockIdx.x * kWarpsPerCta + wid) * kPlaneWords;
    for (;;) {
    int qi = 0;
    if (lane == 0) qi = (int)atomicAdd(queue, 1u);
    qi = __shfl_sync(0xffffffffu, qi, 0);
    if (qi >= njobs) break;
    const int jid = order ? (int)order[qi] : qi;
    const j2k_cb_job J = jobs[jid];
    if (J.cw == 0 || J.ch == 0 || J.cw > 64 || J.ch > 64 || J.orient > 3 || J.sym_cap % 16 != 0) {
        if (lane == 0) {
            atomicCAS(err, 0u, (uint32_t)J2K_DEVERR_BAD_JOB);
            nsyms[jid] = 0;
        }
        continue;
    }
    symbols_of_shape(S, J, jid, lane, coeff, syms, nsyms, pass_end, planes, descs, err, pad);
    }  // queue loop
}

// ---- phase B: MQ encoder ---------------------------------------------------------------------------
//
// The coder is serial per block, so the kernel time is (longest block's symbol count) x (time per
// symbol).  Blocks are ordered longest-first (a radix sort of the symbol counts) so that the blocks of
// a warp pair end together and the biggest ones start first.

__constant__ uint16_t c_qe[47] = {
    0x5601, 0x3401, 0x1801, 0x0AC1, 0x0521, 0x0221, 0x5601, 0x5401, 0x4801, 0x3801, 0x3001, 0x2401,
    0x1C01, 0x1601, 0x5601, 0x5401, 0x5101, 0x4801, 0x3801, 0x3401, 0x3001, 0x2801, 0x2401, 0x2201,
    0x1C01, 0x1801, 0x1601, 0x1401, 0x1201, 0x1101, 0x0AC1, 0x09C1, 0x08A1, 0x0521, 0x0441, 0x02A1,
    0x0221, 0x0141, 0x0111, 0x0085, 0x0049, 0x0025, 0x0015, 0x0009, 0x0005, 0x0001, 0x5601};
__constant__ uint8_t c_nmps[47] = {1,  2,  3,  4,  5,  38, 7,  8,  9,  10, 11, 12, 13, 29, 15, 16,
                                   17, 18, 19, 20, 21, 22, 23, 24, 25, 26, 27, 28, 29, 30, 31, 32,
                                   33, 34, 35, 36, 37, 38, 39, 40, 41, 42, 43, 44, 45, 45, 46};
__constant__ uint8_t c_nlps[47] = {1,  6,  9,  12, 29, 33, 6,  14, 14, 14, 17, 18, 20, 21, 14, 14,
                                   15, 16, 17, 18, 19, 19, 20, 21, 22, 23, 24, 25, 26, 27, 28, 29,
                                   30, 31, 32, 33, 34, 35, 36, 37, 38, 39, 40, 41, 42, 43, 46};

#include "mq_enc.cuh"

constexpr int kMqThreads = 32;  // blocks of a warp pair at most; one pair (64 threads) is a CTA, so that the
                                // longest blocks' pairs spread one per SM

constexpr int kMqCopies = 8;
constexpr int kMqTable = 94 * kMqCopies;

// the 94-entry state table (state * 2 + MPS), each entry kMqCopies times, filled by the threads of
// a CTA
__device__ __forceinline__ void fill_mq_table(MqState* tab) {
    for (int i = threadIdx.x; i < kMqTable; i += blockDim.x) {
        const int k = i / kMqCopies >> 1;
        tab[i] = mq_table_entry(c_qe[k], c_nmps[k], c_nlps[k], k == 0 || k == 6 || k == 14,
                                (uint32_t)(i / kMqCopies & 1));
    }
}
template <int SHIFT>
__device__ __forceinline__ MqMem<SHIFT, kMqCopies> mq_mem(MqState* st, const MqState* tab) {
    return MqMem<SHIFT, kMqCopies>(st, tab + threadIdx.x % kMqCopies);
}
// T.800 Table D.7: the initial states (context k at st[k * stride]; 32 of them, so that a 5-bit
// index needs no clamp)
__device__ __forceinline__ void reset_mq_states(MqState* st, int stride, const MqState* tab) {
    for (int k = 0; k < 32; ++k) st[k * stride] = tab[0];
    st[0] = tab[4 * 2 * kMqCopies];
    st[17 * stride] = tab[3 * 2 * kMqCopies];
    st[18 * stride] = tab[46 * 2 * kMqCopies];
}

// The byte-by-byte MQ encoder registers of the general styled coder, and the byte writer of raw
// passes.
struct MqEnc {
    uint32_t A, C, B;   // B: pending output byte (may still receive a carry)
    int CT, bp;         // bp: index of B (-1 before the first byte)
    uint32_t* out;      // word-aligned codeword buffer
    int cap;            // bytes
    uint32_t wacc;      // completed bytes waiting for a 32-bit store
    int wn, wbase;
    bool ovf;
    __device__ __forceinline__ void push(uint32_t byte) {
        wacc |= byte << (8 * wn);
        if (++wn == 4) {
            if (wbase + 4 <= cap) out[wbase >> 2] = wacc; else ovf = true;
            wbase += 4;
            wn = 0;
            wacc = 0;
        }
    }
    // T.800 C.2 BYTEOUT in one straight-line form: a carry (C >= 2^27 after a non-0xFF byte)
    // increments the pending byte; a 0xFF byte (before or after the carry) is followed by 7 bits.
    __device__ __forceinline__ void byteout() {
        if (B != 0xFF && C >= 0x8000000u) {
            if (bp >= 0) B += 1;
            C &= 0x7FFFFFF;
        }
        const bool ff = (B == 0xFF);
        const uint32_t v = ff ? (C >> 20) : (C >> 19);
        C &= ff ? 0xFFFFFu : 0x7FFFFu;
        CT = ff ? 7 : 8;
        if (bp >= 0) push(B);
        ++bp;
        B = v & 0xFF;
    }
    // shift by sh (0..15) with at most two byte outputs
    __device__ __forceinline__ void renorm(int sh) {
        int k = min(sh, CT);
        A <<= k;
        C <<= k;
        CT -= k;
        sh -= k;
        if (CT == 0) {
            byteout();
            k = min(sh, CT);
            A <<= k;
            C <<= k;
            CT -= k;
            sh -= k;
            if (CT == 0) {
                byteout();
                A <<= sh;
                C <<= sh;
                CT -= sh;
            }
        }
    }
};

// Warp schedule of the MQ kernel: tier k has warps[k] warps of lanes[k] blocks each.
struct MqSchedule {
    int warps[4] = {0, 0, 0, 0};
    int lanes[4] = {0, 0, 0, 0};
};

// Rate control: the bytes made when each bit-plane's cleanup pass ends (pass 3k; pass ends in
// symbols from phase A), into plane_bytes[k].
struct MqPlaneEnds {
    const uint32_t* pe;
    uint32_t* plane_bytes;
    int npasses, k;
    uint32_t end;
    __device__ __forceinline__ void start() {
        k = 0;
        end = npasses > 0 ? pe[0] : 0xFFFFFFFFu;
    }
    __device__ __forceinline__ uint32_t next() const { return end; }
    __device__ __forceinline__ void at(const MqCoder& e) {
        if (k < 32) plane_bytes[k] = (uint32_t)e.cnt;
        ++k;
        end = 3 * k < npasses ? pe[3 * k] : 0xFFFFFFFFu;
    }
};

// Where the two warps of a pair meet, once per chunk in each one's loop.  A numbered barrier, not
// __syncthreads: the meeting places of the two roles are different ones.
__device__ __forceinline__ void mq_pair_barrier() {
    static_assert(kMqThreads == 32, "a pair is 64 threads");
    asm volatile("bar.sync 1, 64;" ::: "memory");
}

// One block per lane of a warp pair (mq_enc.cuh): warp 0 runs the interval part and puts four
// symbols' additions and shifts into a ring in shared memory, warp 1 takes them through the code
// part eight at a time, a chunk of 16 symbols behind.  The two parts are serial chains of their own,
// so a symbol costs the longer one instead of both.  Bound by the interval chain: 33 instructions and
// 67 cycles a symbol for a block alone in its pair (16 symbols unrolled; with four 76), about 90 with
// 32 blocks (145 with the bytes taken out four symbols at a time, when the code warp was the slower
// one; 94 with one copy of the state table, whose banks the lanes shared).  One warp with both parts
// took 104 and 165 cycles; an integer coder with a leading-zero count and a branch to the byte output
// in every symbol's chain over 200.  4096 blocks of a 4096 x 4096 gray image, 32 to a pair: 1.45 ms,
// 2.32 with the bytes taken out by fours, 2.44 with one warp.
// RATE: also record the plane ends (MqPlaneEnds) into plane_bytes[job * 32 + k].
template <bool RATE>
__global__ void __launch_bounds__(2 * kMqThreads)
t1_mq_kernel(const uint8_t* __restrict__ syms, const j2k_cb_job* __restrict__ jobs, const uint32_t* __restrict__ nsyms,
             const uint32_t* __restrict__ order, int njobs, uint8_t* __restrict__ bytes,
             j2k_cb_desc* __restrict__ descs, uint32_t* __restrict__ err, const uint32_t* __restrict__ pend,
             uint32_t* __restrict__ plane_bytes, MqSchedule sched, int lanes) {
    __shared__ MqState tab[kMqTable];
    __shared__ MqState cst[32 * kMqThreads];
    __shared__ uint4 ring[2][4][kMqThreads];  // [chunk parity][group][lane]
    __shared__ float last_a[kMqThreads];
    fill_mq_table(tab);
    const int lane = threadIdx.x & 31;
    // pair w takes blocks in longest-first order: the schedule's tiers first (pairs with fewer
    // blocks each), then `lanes` blocks per pair
    const int w = blockIdx.x;
    int gid = -1, mine = lanes, wbase = 0, gbase = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (gid < 0 && w < wbase + sched.warps[k]) {
            mine = sched.lanes[k];
            gid = gbase + (w - wbase) * mine + lane;
        }
        wbase += sched.warps[k];
        gbase += sched.warps[k] * sched.lanes[k];
    }
    if (gid < 0) gid = gbase + (w - wbase) * lanes + lane;
    const bool live = lane < mine && gid < njobs;
    const int jid = live ? (order ? (int)order[gid] : gid) : 0;
    j2k_cb_job J{};
    if (live) J = jobs[jid];
    const int n = live ? (int)min(nsyms[jid], J.sym_cap) : 0;
    const int chunks = (__reduce_max_sync(0xffffffffu, n) + 15) >> 4;  // the same in both warps
    __syncthreads();
    MqCoder e;
    e.init(reinterpret_cast<uint32_t*>(bytes + J.out_off), (int)J.out_cap);
    if (threadIdx.x < 32) {
        MqState* st = cst + lane;
        reset_mq_states(st, kMqThreads, tab);
        MqSymbols<MqMem<5, kMqCopies>> src(syms + J.sym_off, n, mq_mem<5>(st, tab));
        for (int k = 0; k < chunks; ++k) {
            const uint4 c = src.next(k);
            uint32_t wa = c.x, wb = c.y, wc = c.z, wd = c.w, ev[4];
            const auto put = [&](int j, uint32_t add, uint32_t moved) { ev[j] = add | (moved >> 7); };
            if (16 * k + 16 <= n) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    src.group(e, wa, wb, 4, put);
                    ring[k & 1][q][lane] = make_uint4(ev[0], ev[1], ev[2], ev[3]);
                    wa = wb;
                    wb = wc;
                    wc = wd;
                    wd = src.c0.x;
                }
            } else {
#pragma unroll 1
                for (int q = 0; 16 * k + 4 * q < n; ++q) {
                    src.group(e, wa, wb, n - 16 * k - 4 * q, put);
                    ring[k & 1][q][lane] = make_uint4(ev[0], ev[1], ev[2], ev[3]);
                    wa = wb;
                    wb = wc;
                    wc = wd;
                }
            }
            if (16 * k + 16 >= n) last_a[lane] = e.A;  // (again in every chunk after the last symbol)
            mq_pair_barrier();
        }
        return;
    }
    MqPlaneEnds ends{};
    ends.end = 0xFFFFFFFFu;
    if (RATE && live) {
        ends = MqPlaneEnds{pend + (size_t)jid * 92, plane_bytes + (size_t)jid * 32, descs[jid].npasses, 0, 0};
        ends.start();
        while (ends.next() == 0u) ends.at(e);  // passes with no symbols at all
    }
    for (int k = 0; k < chunks; ++k) {
        mq_pair_barrier();  // chunk k is in the ring; the interval warp goes on with chunk k + 1
#pragma unroll 1
        for (int q = 0; q < 4 && 16 * k + 4 * q < n; q += 2) {
            const int at = 16 * k + 4 * q;
            const uint4 r = ring[k & 1][q][lane];
            uint4 t = ring[k & 1][q + 1][lane];
            if (at + 4 >= n) t = make_uint4(0, 0, 0, 0);  // not written: the block has ended
            const uint32_t ev[8] = {r.x, r.y, r.z, r.w, t.x, t.y, t.z, t.w};
            if ((!RATE || ends.next() > (uint32_t)at + 8u) && e.code8(ev)) continue;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                e.C += ev[j] & 0xFFFFu;
                e.shift((int)(ev[j] >> 16));
                if (RATE)
                    while (ends.next() == (uint32_t)(at + j + 1)) ends.at(e);
            }
        }
    }
    if (!live) return;
    int len = 0;
    if (n > 0) {
        e.A = last_a[lane];
        len = e.flush();
    }
    if (e.ovf || len > (int)J.out_cap) {
        atomicCAS(err, 0u, (uint32_t)J2K_DEVERR_OUT_CAPACITY);
        len = 0;
    }
    descs[jid].length = len;
}

// ---- code-block styles: coding units --------------------------------------------------------
//
// With a code-block style the MQ coder works on units: a run of passes coded serially by one
// lane (context states carried from pass to pass, reset where the style says so, the codeword
// terminated after the passes the style terminates, raw-coded passes written as bits).  When
// the style has both RESET and TERMALL every pass starts from fresh states and a fresh coder,
// so each pass is a unit of its own and the passes of a block code in parallel lanes; otherwise
// a block is one unit.  Unit k of job j is slot j * J2K_PASS_STRIDE + k.  A unit writes its
// segments into a slot of its own (its symbols' range of the symbol buffer, times a factor,
// plus 16 bytes per pass), and a compaction pass then puts each block's units back to back.

__host__ __device__ __forceinline__ bool units_per_pass(int style) {
    return (style & (J2K_CBLK_RESET | J2K_CBLK_TERMALL)) == (J2K_CBLK_RESET | J2K_CBLK_TERMALL);
}

// slot byte offset of the unit that starts at symbol s0 and pass p0 of job j (symbol stream of
// job j at sym_off): slots follow the symbols, so consecutive units never overlap
__device__ __forceinline__ uint64_t seg_slot(uint64_t sym_off, uint32_t s0, int j, int p0, int fac) {
    return (uint64_t)fac * ((sym_off + s0 + 3) & ~(uint64_t)3) + 16ull * ((uint64_t)j * J2K_PASS_STRIDE + p0);
}

// first symbol of pass p of a job whose pass ends are pe: with per-pass units every pass's
// symbols start on a 16-byte boundary (phase A pads them)
__device__ __forceinline__ uint32_t pass_start(const uint32_t* pe, int p, bool per_pass) {
    if (p == 0) return 0u;
    return per_pass ? (pe[p - 1] + 15u) & ~15u : pe[p - 1];
}

// sort keys: symbols of each unit + 1 (0 for slots without a unit); values: slot ids
__global__ void t1_unit_keys_kernel(const j2k_cb_desc* __restrict__ descs, const uint32_t* __restrict__ pend,
                                    int njobs, int style, uint32_t* __restrict__ keys, uint32_t* __restrict__ ids) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= njobs * J2K_PASS_STRIDE) return;
    const int j = i / J2K_PASS_STRIDE, k = i % J2K_PASS_STRIDE;
    const int np = descs[j].npasses;
    const uint32_t* pe = pend + (size_t)j * J2K_PASS_STRIDE;
    uint32_t key = 0;
    if (units_per_pass(style)) {
        // raw passes sort after the MQ ones (bit 31), so that a warp's lanes code alike passes
        if (k < np) key = (pe[k] - pass_start(pe, k, true) + 1u) | (j2k_pass_raw(style, k) ? 0u : 0x80000000u);
    } else if (k == 0 && np > 0) {
        key = pe[np - 1] + 1u;
    }
    keys[i] = key;
    ids[i] = (uint32_t)i;
}

// One lane per unit, units longest first.  ulen[slot] receives the unit's bytes; ends[j *
// stride + p] the unit-relative codeword bytes when pass p ended.
__global__ void __launch_bounds__(128)
t1_mq_units_kernel(const uint8_t* __restrict__ syms, const j2k_cb_job* __restrict__ jobs,
                   const j2k_cb_desc* __restrict__ descs, const uint32_t* __restrict__ pend,
                   const uint32_t* __restrict__ order, const uint32_t* __restrict__ keys, int nslots, int style,
                   int fac, uint8_t* __restrict__ segs, uint32_t* __restrict__ ulen, uint32_t* __restrict__ ends,
                   uint32_t* __restrict__ err) {
    __shared__ uint32_t tab[47];
    __shared__ uint32_t cst[32 * 128];
    for (int i = threadIdx.x; i < 47; i += blockDim.x)
        tab[i] = (uint32_t)c_qe[i] | ((uint32_t)c_nmps[i] << 16) | ((uint32_t)c_nlps[i] << 22) |
                 ((uint32_t)(i == 0 || i == 6 || i == 14) << 28);
    __syncthreads();
    const int gid = blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= nslots || keys[gid] == 0) return;  // keys are sorted: the empty slots come last
    const int u = (int)order[gid];
    const int j = u / J2K_PASS_STRIDE, k = u % J2K_PASS_STRIDE;
    const j2k_cb_job J = jobs[j];
    const int np = descs[j].npasses;
    const bool per_pass = units_per_pass(style);
    const int p0 = per_pass ? k : 0, p1 = per_pass ? k + 1 : np;
    const uint32_t* pe = pend + (size_t)j * J2K_PASS_STRIDE;
    uint32_t* eo = ends + (size_t)j * J2K_PASS_STRIDE;
    const uint32_t s0 = p0 ? pe[p0 - 1] : 0u, s1 = pe[p1 - 1];
    if (s1 > J.sym_cap || s0 > s1) {
        atomicCAS(err, 0u, (uint32_t)J2K_DEVERR_BAD_JOB);
        return;
    }
    const uint64_t base = seg_slot(J.sym_off, s0, j, p0, fac);
    const uint64_t lim = seg_slot(J.sym_off, s1, j, p1, fac);
    uint32_t* st = cst + threadIdx.x;  // context c at st[c * 128]
    auto reset_states = [&]() {
        for (int c = 0; c < 32; ++c) st[c * 128] = tab[0];
        st[0] = tab[4];
        st[17 * 128] = tab[3];
        st[18 * 128] = tab[46];
    };
    reset_states();
    MqEnc e;
    e.out = reinterpret_cast<uint32_t*>(segs + base);
    e.cap = (int)(lim - base);
    e.wacc = 0;
    e.wn = 0;
    e.wbase = 0;
    e.ovf = false;
    // raw coder: bits of the byte being filled, bits left in it, the last completed byte (held
    // back one byte so that a final 0xFF can be dropped)
    uint32_t rc = 0;
    int rct = 8, rpend = -1;
    bool rlastff = false, raw = false;
    auto raw_complete = [&](uint32_t b) {
        if (rpend >= 0) e.push((uint32_t)rpend);
        rpend = (int)b;
        rlastff = b == 0xFF;
        rct = rlastff ? 7 : 8;
        rc = 0;
    };
    const uint8_t* sp = syms + J.sym_off;
    for (int p = p0; p < p1; ++p) {
        if (p > p0 && (style & J2K_CBLK_RESET)) reset_states();
        raw = j2k_pass_raw(style, p);
        if (p == p0 || j2k_pass_terminated(style, p - 1, np)) {  // a new segment
            if (raw) {
                rc = 0;
                rct = 8;
                rpend = -1;
                rlastff = false;
            } else {
                e.A = 0x8000;
                e.C = 0;
                e.B = 0;
                e.CT = 12;
                e.bp = -1;
            }
        }
        const uint32_t a = p ? pe[p - 1] : 0u, b = pe[p];
        uint32_t word = 0;
        for (uint32_t i = a; i < b; ++i) {
            if (i == a || (i & 3) == 0) word = __ldcs(reinterpret_cast<const uint32_t*>(sp + (i & ~3u)));
            const uint32_t sym = (word >> (8 * (i & 3))) & 0xFF;
            if (raw) {
                const uint32_t lab = sym & 31;
                const uint32_t bit = ((sym >> 7) ^ ((lab >= 9 && lab <= 13) ? (sym >> 5) : 0u)) & 1u;
                rc = (rc << 1) | bit;
                if (--rct == 0) raw_complete(rc & 0xFF);
            } else {
                const int cx = (int)(sym & 31);
                const int d = (int)(sym >> 7);
                const uint32_t ent = st[cx * 128];
                const uint32_t qe = ent & 0xFFFF;
                const int mps = (int)(ent >> 31);
                const bool is_mps = d == mps;
                const uint32_t a1 = e.A - qe;
                const bool fast = is_mps && (a1 & 0x8000);
                const bool addc = fast || (is_mps != (a1 < qe));
                e.C += addc ? qe : 0u;
                e.A = addc ? a1 : qe;
                if (!fast) {
                    const int nidx = is_mps ? (ent >> 16) & 63 : (ent >> 22) & 63;
                    const uint32_t nmps = (uint32_t)(mps ^ (!is_mps & (int)((ent >> 28) & 1)));
                    st[cx * 128] = tab[nidx] | (nmps << 31);
                }
                e.renorm(__clz(e.A) - 16);
            }
        }
        if (j2k_pass_terminated(style, p, np)) {
            if (raw) {
                if (rct < (rlastff ? 7 : 8)) raw_complete((rc << rct) & 0xFF);
                if (rpend >= 0 && rpend != 0xFF) e.push((uint32_t)rpend);
                rpend = -1;
            } else {  // FLUSH (T.800 C.2.9); a last byte of 0xFF is dropped
                const uint32_t tempc = e.C + e.A;
                e.C |= 0xFFFF;
                if (e.C >= tempc) e.C -= 0x8000;
                e.C <<= e.CT;
                e.byteout();
                e.C <<= e.CT;
                e.byteout();
                if (e.B != 0xFF) e.push(e.B);
            }
            eo[p] = (uint32_t)(e.wbase + e.wn);
        } else {
            eo[p] = (uint32_t)(e.wbase + e.wn) + (raw ? (rpend >= 0) : (uint32_t)(e.bp + 1 > 0));
        }
    }
    // the last partial word
    uint8_t* bb = segs + base;
    for (int q = 0; q < e.wn; ++q) {
        if (e.wbase + q < e.cap) bb[e.wbase + q] = (uint8_t)(e.wacc >> (8 * q));
        else e.ovf = true;
    }
    if (e.ovf) {
        atomicCAS(err, 0u, (uint32_t)J2K_DEVERR_SEG_CAPACITY);
        ulen[u] = 0;
        return;
    }
    ulen[u] = (uint32_t)(e.wbase + e.wn);
}

// A raw pass (T.800 D.6): its decisions as bits, most significant first; a byte after 0xFF holds
// 7, the partial last byte is padded with 0s, a last 0xFF is dropped.  Returns the bytes written.
__device__ uint32_t raw_pass(const uint8_t* syms, int n, uint8_t* seg, int cap, bool* ovf) {
    MqEnc e;  // (its byte writer)
    e.out = reinterpret_cast<uint32_t*>(seg);
    e.cap = cap;
    e.wacc = 0;
    e.wn = 0;
    e.wbase = 0;
    e.ovf = false;
    uint32_t rc = 0;
    int rct = 8, rpend = -1;
    bool rlastff = false;
    auto complete = [&](uint32_t b) {
        if (rpend >= 0) e.push((uint32_t)rpend);
        rpend = (int)b;
        rlastff = b == 0xFF;
        rct = rlastff ? 7 : 8;
        rc = 0;
    };
    const uint4* sp4 = reinterpret_cast<const uint4*>(syms);
    const int nchunks = (n + 15) >> 4;
    const uint4 z4 = make_uint4(0, 0, 0, 0);
    uint4 c0 = nchunks > 0 ? __ldcs(sp4) : z4;
    uint4 c1 = nchunks > 1 ? __ldcs(sp4 + 1) : z4;
    for (int k = 0; k < nchunks; ++k) {
        const uint4 cur = c0;
        c0 = c1;
        c1 = (k + 2 < nchunks) ? __ldcs(sp4 + k + 2) : z4;
        const uint32_t wv[4] = {cur.x, cur.y, cur.z, cur.w};
        const int m = min(16, n - 16 * k);
        for (int i = 0; i < m; ++i) {
            const uint32_t sym = (wv[i >> 2] >> (8 * (i & 3))) & 0xFF;
            const uint32_t lab = sym & 31;
            const uint32_t bit = ((sym >> 7) ^ ((lab >= 9 && lab <= 13) ? (sym >> 5) : 0u)) & 1u;
            rc = (rc << 1) | bit;
            if (--rct == 0) complete(rc & 0xFF);
        }
    }
    if (rct < (rlastff ? 7 : 8)) complete((rc << rct) & 0xFF);
    if (rpend >= 0 && rpend != 0xFF) e.push((uint32_t)rpend);
    for (int q = 0; q < e.wn; ++q) {
        if (e.wbase + q < e.cap) seg[e.wbase + q] = (uint8_t)(e.wacc >> (8 * q));
        else e.ovf = true;
    }
    *ovf = e.ovf;
    return (uint32_t)(e.wbase + e.wn);
}

// Per-pass units (RESET | TERMALL: every pass a codeword segment that starts from fresh context
// states and a fresh coder): one lane per pass, passes longest first, the MQ passes before the
// raw ones.  An MQ pass runs the same loop as t1_mq_kernel (mq_enc.cuh), from its 16-byte aligned
// start, and ends with the FLUSH of T.800 C.2.9 (a last 0xFF dropped), however few symbols it has;
// a raw pass writes its decisions as bits (raw_pass).
// Unit bytes go to the pass's slot; ulen / ends as t1_mq_units_kernel.
constexpr int kPassThreads = 128;
static_assert(kMqThreads == 1 << 5 && kPassThreads == 1 << 7, "MqMem strides");

__global__ void __launch_bounds__(kPassThreads)
t1_mq_pass_kernel(const uint8_t* __restrict__ syms, const j2k_cb_job* __restrict__ jobs,
                  const j2k_cb_desc* __restrict__ descs, const uint32_t* __restrict__ pend,
                  const uint32_t* __restrict__ order, const uint32_t* __restrict__ keys, int nslots, int style,
                  int fac, uint8_t* __restrict__ segs, uint32_t* __restrict__ ulen, uint32_t* __restrict__ ends,
                  uint32_t* __restrict__ err) {
    __shared__ MqState tab[kMqTable];
    __shared__ MqState cst[32 * kPassThreads];
    fill_mq_table(tab);
    __syncthreads();
    const int gid = blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= nslots || keys[gid] == 0) return;  // keys are sorted: the empty slots come last
    const int u = (int)order[gid];
    const int j = u / J2K_PASS_STRIDE, p = u % J2K_PASS_STRIDE;
    const j2k_cb_job J = jobs[j];
    const uint32_t* pe = pend + (size_t)j * J2K_PASS_STRIDE;
    const uint32_t s0 = pass_start(pe, p, true), s1 = pe[p];
    const uint32_t snext = (s1 + 15u) & ~15u;  // where the next pass's symbols (and slot) start
    if (s1 > J.sym_cap || s0 > s1) {
        atomicCAS(err, 0u, (uint32_t)J2K_DEVERR_BAD_JOB);
        return;
    }
    const int n = (int)(s1 - s0);
    const uint64_t base = seg_slot(J.sym_off, s0, j, p, fac);
    const uint64_t lim = seg_slot(J.sym_off, snext, j, p + 1, fac);
    uint32_t len;
    bool ovf;
    if (j2k_pass_raw(style, p)) {
        len = raw_pass(syms + J.sym_off + s0, n, segs + base, (int)(lim - base), &ovf);
    } else {
        MqState* st = cst + threadIdx.x;
        reset_mq_states(st, kPassThreads, tab);
        MqCoder e;
        e.init(reinterpret_cast<uint32_t*>(segs + base), (int)(lim - base));
        mq_encode(e, syms + J.sym_off + s0, n, mq_mem<7>(st, tab));
        len = (uint32_t)e.flush();
        ovf = e.ovf;
    }
    if (ovf) {
        atomicCAS(err, 0u, (uint32_t)J2K_DEVERR_SEG_CAPACITY);
        ulen[u] = 0;
        return;
    }
    ulen[u] = len;
    ends[(size_t)j * J2K_PASS_STRIDE + p] = len;
}

// One warp per code-block: its units' segments back to back into the block's codeword, the
// pass ends made block-relative, and the descriptor's length.
__global__ void t1_units_compact_kernel(const j2k_cb_job* __restrict__ jobs, j2k_cb_desc* __restrict__ descs,
                                        const uint32_t* __restrict__ pend, int njobs, int style, int fac,
                                        const uint8_t* __restrict__ segs, const uint32_t* __restrict__ ulen,
                                        uint32_t* __restrict__ ends, uint8_t* __restrict__ bytes,
                                        uint32_t* __restrict__ err) {
    const int j = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (j >= njobs) return;
    const j2k_cb_job J = jobs[j];
    const int np = descs[j].npasses;
    const bool per_pass = units_per_pass(style);
    const int nu = np == 0 ? 0 : (per_pass ? np : 1);
    const uint32_t* pe = pend + (size_t)j * J2K_PASS_STRIDE;
    uint32_t* eo = ends + (size_t)j * J2K_PASS_STRIDE;
    uint32_t run = 0;  // bytes of the units before this round of 32
    uint8_t* dst = bytes + J.out_off;
    for (int k0 = 0; k0 < nu; k0 += 32) {
        const int k = k0 + lane;
        const uint32_t len = k < nu ? ulen[(size_t)j * J2K_PASS_STRIDE + k] : 0u;
        int tot;
        const uint32_t off = run + (uint32_t)warp_excl((int)len, lane, &tot);
        if (k < nu) {
            if (off + len > J.out_cap) {
                atomicCAS(err, 0u, (uint32_t)J2K_DEVERR_OUT_CAPACITY);
            } else {
                const int p0 = per_pass ? k : 0, p1 = per_pass ? k + 1 : np;
                for (int p = p0; p < p1; ++p) eo[p] += off;
            }
        }
        // the round's units copied one after another, each by the whole warp
        const bool ok = k < nu && off + len <= J.out_cap;
        const unsigned okm = __ballot_sync(0xffffffffu, ok);
        for (int q = 0; q < 32; ++q) {
            if (!((okm >> q) & 1u)) continue;
            const uint32_t ql = __shfl_sync(0xffffffffu, len, q), qo = __shfl_sync(0xffffffffu, off, q);
            const int kq = k0 + q;
            const int p0 = per_pass ? kq : 0;
            const uint8_t* src = segs + seg_slot(J.sym_off, pass_start(pe, p0, per_pass), j, p0, fac);
            for (uint32_t b = (uint32_t)lane; b < ql; b += 32) dst[qo + b] = src[b];
        }
        run += (uint32_t)tot;
    }
    for (int p = np + lane; p < J2K_PASS_STRIDE; p += 32) eo[p] = 0;
    if (lane == 0) descs[j].length = run <= J.out_cap ? (int32_t)run : 0;
}

__global__ void iota_kernel(uint32_t* v, int n) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) v[i] = (uint32_t)i;
}

// Squared reconstruction error of every code-block when decoded down to bit-plane k only
// (dist[job * 33 + k]; magnitudes below the last decoded plane at the middle of their interval)
// and with nothing decoded (dist[job * 33 + 32]).  One warp per block, kDistWarps blocks per CTA.
// Each lane keeps one exact 64-bit sum per plane p in registers: a sample of magnitude m with
// top bit b adds its midpoint error at the planes p <= b and m^2 at the planes above b; the
// lanes' sums are then added by shuffles.  Integer sums, so the result (and the truncation
// choices built on it) does not depend on the order of the additions.
constexpr int kDistWarps = 4;
__global__ void __launch_bounds__(kDistWarps * 32)
t1_dist_kernel(const int32_t* __restrict__ coeff, const j2k_cb_job* __restrict__ jobs,
               const j2k_cb_desc* __restrict__ descs, int njobs, double* __restrict__ dist) {
    const int lane = threadIdx.x & 31;
    const int jid = blockIdx.x * kDistWarps + (threadIdx.x >> 5);
    if (jid >= njobs) return;
    const j2k_cb_job J = jobs[jid];
    const int nb = min((int)descs[jid].numbps, 31);  // the same for the whole warp
    unsigned long long acc[31], total = 0;
#pragma unroll
    for (int p = 0; p < 31; ++p) acc[p] = 0;
    if (J.cw <= 64 && J.ch <= 64) {
        for (int y = 0; y < J.ch; ++y) {
            const int32_t* row = coeff + J.off + (size_t)y * J.pitch;
            for (int x = lane; x < J.cw; x += 32) {
                const int32_t v = row[x];
                const uint32_t m = v < 0 ? (uint32_t)(-(int64_t)v) : (uint32_t)v;
                const int b = 31 - __clz(m);  // -1 for m = 0, which adds nothing
                const unsigned long long m2 = (unsigned long long)m * m;
                total += m2;
#pragma unroll
                for (int p = 0; p < 31; ++p) {
                    if (p >= nb) break;
                    // m - (m truncated to plane p + half its interval); |e| < 2^30
                    const int e = (int)(m & ((1u << p) - 1u)) - (int)((1u << p) >> 1);
                    acc[p] += p <= b ? (unsigned long long)((long long)e * e) : m2;
                }
            }
        }
    }
#pragma unroll
    for (int p = 0; p < 31; ++p) {
        if (p >= nb) break;
        unsigned long long s = acc[p];
        for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        acc[p] = s;
    }
    for (int o = 16; o; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
    if (lane == 0) {
        double* d = dist + (size_t)jid * 33;
        // plane p is the last decoded one after k = nb - 1 - p planes
#pragma unroll
        for (int p = 0; p < 31; ++p)
            if (p < nb) d[nb - 1 - p] = (double)acc[p];
        for (int k = nb; k < 32; ++k) d[k] = 0.0;
        d[32] = (double)total;
    }
}

}  // namespace

// Phase B of a styled encode: units keyed and sorted longest first, coded one lane each, then
// compacted into the blocks' codewords.
static j2k_status encode_styled_units(j2k_ctx* ctx, const j2k_cb_job* d_jobs, size_t njobs, j2k_cb_desc* descs,
                                      uint8_t* bytes, size_t sym_bytes, const uint8_t* syms, const uint32_t* pend,
                                      int style, uint32_t* pass_ends, cudaStream_t st) {
    const size_t nslots = njobs * J2K_PASS_STRIDE;
    if (nslots > 0x7FFFFFFF) return j2k_fail(ctx, J2K_ERR_UNSUPPORTED, "too many code-blocks for a styled encode");
    uint32_t* ub = (uint32_t*)j2k_scratch(ctx, SCR_UNITS, (nslots * (pass_ends ? 5 : 6) + 64) * 4);
    if (!ub) return J2K_ERR_OUT_OF_MEMORY;
    uint32_t* keys_in = ub;
    uint32_t* keys_out = keys_in + nslots;
    uint32_t* ids_in = keys_out + nslots;
    uint32_t* ids_out = ids_in + nslots;
    uint32_t* ulen = ids_out + nslots;
    uint32_t* ends = pass_ends ? pass_ends : ulen + nslots;
    const int fac = std::max(1, ctx->t1_seg_factor);
    // slots end by fac * (sym_bytes + 3) + 16 * nslots (seg_slot of the last unit's end)
    uint8_t* segs = (uint8_t*)j2k_scratch(ctx, SCR_SEGS, (size_t)fac * (sym_bytes + 64) + 16 * nslots + 64);
    if (!segs) return J2K_ERR_OUT_OF_MEMORY;
    const unsigned g = (unsigned)((nslots + 255) / 256);
    t1_unit_keys_kernel<<<g, 256, 0, st>>>(descs, pend, (int)njobs, style, keys_in, ids_in);
    J2K_CUDA(ctx, cudaGetLastError());
    size_t tmp = 0;
    cub::DeviceRadixSort::SortPairsDescending(nullptr, tmp, keys_in, keys_out, ids_in, ids_out, (int)nslots, 0, 32,
                                              st);
    void* tbuf = j2k_scratch(ctx, SCR_MISC, tmp + 16);
    if (!tbuf) return J2K_ERR_OUT_OF_MEMORY;
    J2K_CUDA(ctx, cub::DeviceRadixSort::SortPairsDescending(tbuf, tmp, keys_in, keys_out, ids_in, ids_out,
                                                            (int)nslots, 0, 32, st));
    if (units_per_pass(style))
        t1_mq_pass_kernel<<<(unsigned)((nslots + kPassThreads - 1) / kPassThreads), kPassThreads, 0, st>>>(
            syms, d_jobs, descs, pend, ids_out, keys_out, (int)nslots, style, fac, segs, ulen, ends, ctx->d_err);
    else
        t1_mq_units_kernel<<<(unsigned)((nslots + 127) / 128), 128, 0, st>>>(syms, d_jobs, descs, pend, ids_out,
                                                                             keys_out, (int)nslots, style, fac, segs,
                                                                             ulen, ends, ctx->d_err);
    J2K_CUDA(ctx, cudaGetLastError());
    t1_units_compact_kernel<<<(unsigned)((njobs * 32 + 255) / 256), 256, 0, st>>>(
        d_jobs, descs, pend, (int)njobs, style, fac, segs, ulen, ends, bytes, ctx->d_err);
    J2K_CUDA(ctx, cudaGetLastError());
    return J2K_OK;
}

// Rate control also needs the distortion of each truncation point (the coefficients are still in
// place); the MQ coder has recorded the byte positions at every bit-plane end.
static j2k_status launch_dist(j2k_ctx* ctx, const int32_t* coeff, const j2k_cb_job* d_jobs, const j2k_cb_desc* descs,
                              size_t njobs, double* dist, cudaStream_t st) {
    t1_dist_kernel<<<(unsigned)((njobs + kDistWarps - 1) / kDistWarps), kDistWarps * 32, 0, st>>>(coeff, d_jobs, descs,
                                                                                                 (int)njobs, dist);
    J2K_CUDA(ctx, cudaGetLastError());
    return J2K_OK;
}

j2k_status j2k_t1_encode_jobs(j2k_ctx* ctx, const int32_t* coeff, const j2k_cb_job* d_jobs, size_t njobs,
                              j2k_cb_desc* descs, uint8_t* bytes, size_t sym_bytes,
                              const uint32_t* d_order, cudaStream_t st, uint32_t* plane_bytes, double* dist,
                              int style, uint32_t* pass_ends) {
    if (njobs == 0) return J2K_OK;
    if (style && (plane_bytes || dist))
        return j2k_fail(ctx, J2K_ERR_UNSUPPORTED, "rate control with a code-block style");
    if (((uintptr_t)bytes & 15) != 0)
        return j2k_fail(ctx, J2K_ERR_INVALID_ARG, "t1: bytes buffer must be 16-byte aligned");
    uint8_t* syms = (uint8_t*)j2k_scratch(ctx, SCR_SYMS, sym_bytes + 64);
    // persistent phase A: one bit-plane slot per resident warp
    int per_sm = 0;
    const auto symbols = ctx->t1a_ctas == 3 ? t1_symbols_kernel<3> : t1_symbols_kernel<2>;
    constexpr size_t sym_smem = kWarpsPerCta * sizeof(SymSmem);
    J2K_CUDA(ctx, cudaFuncSetAttribute(symbols, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sym_smem));
    J2K_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, symbols, kWarpsPerCta * 32, sym_smem));
    per_sm = std::max(per_sm, 1);
    const size_t ctas = std::min<size_t>((njobs + kWarpsPerCta - 1) / kWarpsPerCta, (size_t)per_sm * ctx->sm_count);
    uint64_t* planes = (uint64_t*)j2k_scratch(ctx, SCR_PLANES, ctas * kWarpsPerCta * kPlaneWords * 8 + 64);
    // meta: queue head | nsyms | pass ends (92 per job) | sort keys/values (3 arrays of njobs)
    size_t meta_words = 16 + njobs * (1 + 92 + 3) + 64;
    uint32_t* meta = (uint32_t*)j2k_scratch(ctx, SCR_T1STATE, meta_words * 4);
    if (!syms || !meta || !planes) return J2K_ERR_OUT_OF_MEMORY;
    uint32_t* queue = meta;
    uint32_t* nsyms = meta + 16;
    uint32_t* pend = nsyms + njobs;
    uint32_t* keys_out = pend + njobs * 92;
    uint32_t* idx_in = keys_out + njobs;
    uint32_t* idx_out = idx_in + njobs;
    J2K_CUDA(ctx, cudaMemsetAsync(queue, 0, 4, st));
    // with per-pass coding units (RESET | TERMALL) every pass's symbols start 16-byte aligned
    const int pad = (style & (J2K_CBLK_RESET | J2K_CBLK_TERMALL)) == (J2K_CBLK_RESET | J2K_CBLK_TERMALL) ? 1 : 0;
    symbols<<<(unsigned)ctas, kWarpsPerCta * 32, sym_smem, st>>>(coeff, d_jobs, (int)njobs, d_order, queue, syms, nsyms,
                                                                 pend, planes, descs, ctx->d_err, pad);
    J2K_CUDA(ctx, cudaGetLastError());
    if (style)
        return encode_styled_units(ctx, d_jobs, njobs, descs, bytes, sym_bytes, syms, pend, style, pass_ends, st);
    // longest-first order for the MQ lanes
    iota_kernel<<<(unsigned)((njobs + 255) / 256), 256, 0, st>>>(idx_in, (int)njobs);
    size_t tmp = 0;
    cub::DeviceRadixSort::SortPairsDescending(nullptr, tmp, nsyms, keys_out, idx_in, idx_out, (int)njobs, 0, 32, st);
    void* tbuf = j2k_scratch(ctx, SCR_MISC, tmp + 16);
    if (!tbuf) return J2K_ERR_OUT_OF_MEMORY;
    J2K_CUDA(ctx, cub::DeviceRadixSort::SortPairsDescending(tbuf, tmp, nsyms, keys_out, idx_in, idx_out,
                                                            (int)njobs, 0, 32, st));
    const bool rate = plane_bytes && dist;
    // tiers of the schedule, cut to the blocks there are
    MqSchedule sc{};
    size_t left = njobs, warps = 0;
    for (int k = 0; k < J2K_MQ_TIERS && ctx->mq_tier_lanes[k] > 0 && left > 0; ++k) {
        const size_t l = (size_t)ctx->mq_tier_lanes[k];
        const size_t wk = std::min<size_t>((size_t)ctx->mq_tier_warps[k], (left + l - 1) / l);
        sc.warps[k] = (int)wk;
        sc.lanes[k] = (int)l;
        left -= std::min(left, wk * l);
        warps += wk;
    }
    // blocks per pair after the tiers: one more pair per SM holds the rest (a scheduler for each of
    // the warps of two pairs per SM), up to full warps.  Whole lossless encodes of colour images on
    // B200 after a tier of one block per SM, by this rule / with 8 / 16 / 32 a pair: 777 blocks (5 a
    // pair) 1.51 ms with any of them; 1749 (11) 1.56 / 1.78 / 1.56 / 1.58; 3072 (20) 1.69 / 1.95 /
    // 1.94 / 1.73; 5511 (32) 2.17 / 2.88 / 2.23 / 2.17; 12288 (32) 2.77 / 5.18 / 3.94 / 2.78
    const size_t per = (size_t)ctx->sm_count;
    const int lanes = ctx->mq_lanes ? ctx->mq_lanes : (int)std::min<size_t>(std::max<size_t>((left + per - 1) / per, 1), 32);
    warps += (left + lanes - 1) / lanes;
    const auto mq = rate ? t1_mq_kernel<true> : t1_mq_kernel<false>;
    mq<<<(unsigned)warps, 2 * kMqThreads, 0, st>>>(syms, d_jobs, nsyms, idx_out, (int)njobs, bytes, descs, ctx->d_err, pend,
                                               plane_bytes, sc, lanes);
    J2K_CUDA(ctx, cudaGetLastError());
    return rate ? launch_dist(ctx, coeff, d_jobs, descs, njobs, dist, st) : J2K_OK;
}
