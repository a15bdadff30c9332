// The MQ encoder of the device kernels (csrc/mq_enc.cuh), run on the CPU against the flowcharts of
// T.800 Annex C.2 written out bit by bit: random contexts, decisions of every skew, streams of 0 to
// 20000 symbols (all remainders of a group of four).  Byte 0xFF followed by a late carry, which the
// group coder codes again, is met thousands of times.  Prints "streams N symbols M" and exits 0.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

#include "mq_enc.cuh"

static const uint16_t QE[47] = {
    0x5601, 0x3401, 0x1801, 0x0AC1, 0x0521, 0x0221, 0x5601, 0x5401, 0x4801, 0x3801, 0x3001, 0x2401,
    0x1C01, 0x1601, 0x5601, 0x5401, 0x5101, 0x4801, 0x3801, 0x3401, 0x3001, 0x2801, 0x2401, 0x2201,
    0x1C01, 0x1801, 0x1601, 0x1401, 0x1201, 0x1101, 0x0AC1, 0x09C1, 0x08A1, 0x0521, 0x0441, 0x02A1,
    0x0221, 0x0141, 0x0111, 0x0085, 0x0049, 0x0025, 0x0015, 0x0009, 0x0005, 0x0001, 0x5601};
static const uint8_t NMPS[47] = {1,  2,  3,  4,  5,  38, 7,  8,  9,  10, 11, 12, 13, 29, 15, 16,
                                 17, 18, 19, 20, 21, 22, 23, 24, 25, 26, 27, 28, 29, 30, 31, 32,
                                 33, 34, 35, 36, 37, 38, 39, 40, 41, 42, 43, 44, 45, 45, 46};
static const uint8_t NLPS[47] = {1,  6,  9,  12, 29, 33, 6,  14, 14, 14, 17, 18, 20, 21, 14, 14,
                                 15, 16, 17, 18, 19, 19, 20, 21, 22, 23, 24, 25, 26, 27, 28, 29,
                                 30, 31, 32, 33, 34, 35, 36, 37, 38, 39, 40, 41, 42, 43, 46};
static bool switches(int i) { return i == 0 || i == 6 || i == 14; }

struct Flowchart {  // T.800 C.2.2 to C.2.9
    uint32_t A = 0x8000, C = 0;
    int CT = 12, I[19] = {}, MPS[19] = {};
    std::vector<uint8_t> b;
    void put(bool stuffed) {
        b.push_back((uint8_t)(C >> (stuffed ? 20 : 19)));
        C &= stuffed ? 0xFFFFF : 0x7FFFF;
        CT = stuffed ? 7 : 8;
    }
    void byteout() {
        if (!b.empty() && b.back() == 0xFF) return put(true);
        if (C < 0x8000000) return put(false);
        C &= 0x7FFFFFF;
        if (!b.empty()) b.back()++;
        put(!b.empty() && b.back() == 0xFF);
    }
    void renorm() {
        do {
            A = (A << 1) & 0xFFFF;
            C <<= 1;
            if (--CT == 0) byteout();
        } while (!(A & 0x8000));
    }
    void code(int cx, int d) {
        const int i = I[cx];
        const uint32_t q = QE[i];
        A -= q;
        if (d == MPS[cx]) {
            if (A & 0x8000) {
                C += q;
                return;
            }
            if (A < q) A = q;
            else C += q;
            I[cx] = NMPS[i];
        } else {
            if (A < q) C += q;
            else A = q;
            if (switches(i)) MPS[cx] ^= 1;
            I[cx] = NLPS[i];
        }
        renorm();
    }
    void flush() {
        const uint32_t t = C + A;
        C |= 0xFFFF;
        if (C >= t) C -= 0x8000;
        C <<= CT;
        byteout();
        C <<= CT;
        byteout();
        if (!b.empty() && b.back() == 0xFF) b.pop_back();
    }
};

int main(int argc, char** argv) {
    const int streams = argc > 1 ? std::atoi(argv[1]) : 1000;
    std::mt19937_64 rng(7);
    MqState tab[94];
    for (int i = 0; i < 94; ++i)
        tab[i] = mq_table_entry(QE[i >> 1], NMPS[i >> 1], NLPS[i >> 1], switches(i >> 1), i & 1);
    std::vector<uint32_t> out(16384);
    long symbols = 0;
    for (int it = 0; it < streams; ++it) {
        const int n = it % 50 == 0 ? 20000 : (int)(rng() % 600), nctx = 1 + (int)(rng() % 19), mode = (int)(rng() % 4);
        double p = mode == 1 ? 0.001 : (mode == 2 ? 0.5 : (rng() % 1000) / 1000.0);
        std::vector<uint4> words((n + 47) / 16);
        uint8_t* sym = reinterpret_cast<uint8_t*>(words.data());
        for (size_t i = 0; i < words.size() * 16; ++i) sym[i] = (uint8_t)rng();  // past the end: anything
        for (int i = 0; i < n; ++i) {
            if (mode == 3 && rng() % 40 == 0) p = (rng() % 1000) / 1000.0;
            const int d = (rng() % 100000) / 100000.0 < p;
            sym[i] = (uint8_t)(rng() % nctx | (unsigned)d << 7 | (unsigned)(rng() & 1) << 5);
        }
        Flowchart f;
        f.I[0] = 4;
        f.I[17] = 3;
        f.I[18] = 46;
        for (int i = 0; i < n; ++i) f.code(sym[i] & 31, sym[i] >> 7);
        if (n) f.flush();
        MqState st[32];
        for (auto& s : st) s = tab[0];
        st[0] = tab[8];
        st[17] = tab[6];
        st[18] = tab[92];
        MqCoder e;
        e.init(out.data(), (int)out.size() * 4);
        mq_encode(e, sym, n, MqMem<0>(st, tab));
        const int len = n ? e.flush() : 0;
        if (e.ovf || len != (int)f.b.size() || std::memcmp(out.data(), f.b.data(), (size_t)len) != 0) {
            std::printf("stream %d of %d symbols differs\n", it, n);
            return 1;
        }
        // the same as the device's warp pair does it: all intervals first, then eight symbols at a time
        for (auto& x : st) x = tab[0];
        st[0] = tab[8];
        st[17] = tab[6];
        st[18] = tab[92];
        MqCoder iv, cd;
        iv.init(nullptr, 0);
        cd.init(out.data(), (int)out.size() * 4);
        std::fill(out.begin(), out.begin() + f.b.size() / 4 + 1, 0u);
        std::vector<uint32_t> ev(n + 16, 0);
        MqSymbols<MqMem<0>> src(sym, n, MqMem<0>(st, tab));
        for (int k = 0; k < src.nchunks; ++k) {
            const uint4 c = src.next(k);
            const uint32_t w[5] = {c.x, c.y, c.z, c.w, src.c0.x};
            for (int q = 0; q < 4 && 16 * k + 4 * q < n; ++q)
                src.group(iv, w[q], w[q + 1], std::min(4, n - 16 * k - 4 * q),
                          [&](int j, uint32_t add, uint32_t moved) { ev[16 * k + 4 * q + j] = add | (moved >> 7); });
        }
        for (int i = 0; i < n; i += 8) {
            const uint32_t e8[8] = {ev[i], ev[i + 1], ev[i + 2], ev[i + 3], ev[i + 4], ev[i + 5], ev[i + 6], ev[i + 7]};
            if (!cd.code8(e8)) cd.code_each(e8);
        }
        cd.A = iv.A;
        const int len2 = n ? cd.flush() : 0;
        if (cd.ovf || len2 != (int)f.b.size() || std::memcmp(out.data(), f.b.data(), (size_t)len2) != 0) {
            std::printf("stream %d of %d symbols differs by eights\n", it, n);
            return 1;
        }
        symbols += n;
    }
    std::printf("streams %d symbols %ld\n", streams, symbols);
    return 0;
}
