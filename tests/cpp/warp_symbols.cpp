// The context modelling of one code-block (csrc/t1sym.cuh, a warp's work) run on the CPU, a host
// thread per lane.  The warp intrinsics are built to what CUDA promises of them and no more:
// __syncwarp orders the lanes' memory accesses, shuffles, votes and reductions only exchange values
// (relaxed atomics, which ThreadSanitizer takes for no ordering).  Compiled with -fsanitize=thread,
// any two lanes' accesses of shared or global memory that only a shuffle separates are reported.
//
// Reads code-blocks from standard input (cw, ch, orient, pad as int32, then cw * ch int32 samples)
// until its end and writes for each: the number of symbols (int32), then the symbols, the padding of
// passes left out.
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <thread>
#include <vector>

#include <sched.h>

#include "j2k_internal.cuh"

#ifndef __noinline__
#define __noinline__ __attribute__((noinline))
#endif

namespace {

struct Meeting {  // of 32 threads
    std::atomic<int> arrived{0}, round{0};
    void meet(std::memory_order arrive, std::memory_order pass, std::memory_order leave) {
        const int r = round.load(std::memory_order_relaxed);
        if (arrived.fetch_add(1, arrive) == 31) {
            arrived.store(0, std::memory_order_relaxed);
            round.fetch_add(1, pass);
        } else {
            while (round.load(leave) == r) sched_yield();
        }
    }
};
Meeting value_meeting, order_meeting;
std::atomic<uint64_t> slots[2][32];
thread_local int my_lane = 0, values = 0;

// every lane's value, in all[]
void exchange(uint64_t v, uint64_t (&all)[32]) {
    auto& s = slots[values++ & 1];
    s[my_lane].store(v, std::memory_order_relaxed);
    value_meeting.meet(std::memory_order_relaxed, std::memory_order_relaxed, std::memory_order_relaxed);
    for (int i = 0; i < 32; ++i) all[i] = s[i].load(std::memory_order_relaxed);
}
void __syncwarp() {
    order_meeting.meet(std::memory_order_acq_rel, std::memory_order_release, std::memory_order_acquire);
}
template <class T>
T lane_value(T v, int src) {
    uint64_t all[32];
    exchange((uint64_t)v, all);
    return src < 0 || src > 31 ? v : (T)all[src];
}
template <class T>
T __shfl_sync(unsigned, T v, int src) { return lane_value(v, src & 31); }
template <class T>
T __shfl_up_sync(unsigned, T v, int d) { return lane_value(v, my_lane - d); }
template <class T>
T __shfl_down_sync(unsigned, T v, int d) { return lane_value(v, my_lane + d); }
unsigned __ballot_sync(unsigned, bool p) {
    uint64_t all[32];
    exchange(p, all);
    unsigned m = 0;
    for (int i = 0; i < 32; ++i) m |= (unsigned)all[i] << i;
    return m;
}
bool __any_sync(unsigned m, bool p) { return __ballot_sync(m, p) != 0; }
uint32_t __reduce_or_sync(unsigned, uint32_t v) {
    uint64_t all[32];
    exchange(v, all);
    uint32_t m = 0;
    for (uint64_t a : all) m |= (uint32_t)a;
    return m;
}
int __popc(uint32_t x) { return __builtin_popcount(x); }
int __ffs(int x) { return __builtin_ffs(x); }
int __clz(uint32_t x) { return x ? __builtin_clz(x) : 32; }
uint32_t __funnelshift_l(uint32_t lo, uint32_t hi, int s) { return (uint32_t)((((uint64_t)hi << 32 | lo) << s) >> 32); }
uint32_t __funnelshift_r(uint32_t lo, uint32_t hi, int s) { return (uint32_t)(((uint64_t)hi << 32 | lo) >> s); }
uint32_t __byte_perm(uint32_t a, uint32_t b, uint32_t sel) {
    const uint64_t v = (uint64_t)b << 32 | a;
    uint32_t r = 0;
    for (int i = 0; i < 4; ++i) r |= (uint32_t)((v >> (8 * ((sel >> (4 * i)) & 7))) & 255u) << (8 * i);
    return r;
}
void atomicCAS(uint32_t* p, uint32_t, uint32_t v) { *p = v; }

int warp_excl(int v, int lane, int* tot) {
    uint64_t all[32];
    exchange((uint64_t)v, all);
    int before = 0;
    *tot = 0;
    for (int i = 0; i < 32; ++i) {
        if (i < lane) before += (int)all[i];
        *tot += (int)all[i];
    }
    return before;
}

#include "t1sym.cuh"

}  // namespace

int main() {
    int32_t head[4];
    while (std::fread(head, 4, 4, stdin) == 4) {
        const int cw = head[0], ch = head[1], pad = head[3];
        std::vector<int32_t> coeff((size_t)cw * ch);
        if (std::fread(coeff.data(), 4, coeff.size(), stdin) != coeff.size()) return 2;
        j2k_cb_job J{};
        J.pitch = (uint32_t)cw;
        J.cw = (uint16_t)cw;
        J.ch = (uint16_t)ch;
        J.orient = (uint8_t)head[2];
        J.sym_cap = (uint32_t)((cw * ch * 70 + 92 * 16 + 64) / 16 * 16);
        std::vector<uint4> syms(J.sym_cap / 16);
        std::vector<uint64_t> planes(64 * 32);
        std::vector<uint32_t> pend(92);
        uint32_t nsyms = 0, err = 0;
        j2k_cb_desc d{};
        auto smem = std::make_unique<SymSmem>();
        uint8_t* out = reinterpret_cast<uint8_t*>(syms.data());
        std::vector<std::thread> lanes;
        for (int lane = 0; lane < 32; ++lane)
            lanes.emplace_back([&, lane] {
                my_lane = lane;
                symbols_of_shape(*smem, J, 0, lane, coeff.data(), out, &nsyms, pend.data(), planes.data(), &d, &err,
                                 pad);
            });
        for (auto& t : lanes) t.join();
        if (err) return 3;
        std::vector<uint8_t> s;
        uint32_t at = 0;
        for (int p = 0; p < d.npasses; ++p) {
            s.insert(s.end(), out + at, out + pend[p]);
            at = pad ? (pend[p] + 15u) & ~15u : pend[p];
        }
        if (at != nsyms) return 4;
        const int32_t n = (int32_t)s.size();
        std::fwrite(&n, 4, 1, stdout);
        std::fwrite(s.data(), 1, s.size(), stdout);
    }
    return 0;
}
