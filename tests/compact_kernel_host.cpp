// dfs_compact_kernel (csrc/emp_btc.cu) on the CPU: the kernel's own source, compiled for the host,
// one user context per lane, which change places at the warp's collectives; one block of 128 lanes,
// its memory plain host memory.  Every read of the tables in global memory is checked.  Used by
// test_compact_kernel_cpu.py.  Standard input:
//   tables_in_smem min_nw budget capacity deadline stop_at_first stop_at_any
//   puzzles, then per puzzle: width height 4 * width * height colours
//   records, then per record: puzzle length transitions
// deadline counts the clock, which ticks once a warp collective (0: none).  Prints per puzzle
// "nodes solutions incomplete", then "end <clock> rounds <rounds> full <rounds with a full queue>".
#include "emp_bt.h"
#include "emp_compact.h"
#include "emp_model.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <csetjmp>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <ucontext.h>
#include <utility>
#include <vector>

namespace {

constexpr uint32_t kThreads = 128;

struct Warp {
    uint64_t value[2][32];
    uint32_t arrived = 0, phase = 0;
    uint64_t some[32];  // a collective of some of the lanes
    unsigned peers[32];
    uint32_t some_arrived = 0, some_phase = 0;
};
struct Lane {
    ucontext_t first;
    jmp_buf at;
    bool started = false, done = false;
    std::vector<char> stack = std::vector<char>(256 * 1024);
};

Warp g_warps[kThreads / 32];
Lane g_lanes[kThreads];
uint32_t g_block_arrived = 0, g_block_phase = 0;
uint32_t g_tid = 0;
jmp_buf g_scheduler;
unsigned long long g_clock = 0;

struct Tables {  // from and to where the 16-byte records, the 16-bit entries and all of a blob lie
    const char *quads[2], *entries[2], *all[2];
};
std::vector<Tables> g_tables;

__attribute__((noinline)) void yield()
{
    const uint32_t me = g_tid;
    if (!_setjmp(g_lanes[me].at)) _longjmp(g_scheduler, 1);
}

// every lane of the warp leaves a value; returns all of them
const uint64_t* exchange(uint64_t v)
{
    Warp& w = g_warps[g_tid / 32];
    const uint32_t phase = w.phase;
    w.value[phase & 1u][g_tid % 32] = v;
    if (++w.arrived == 32) {
        w.arrived = 0;
        ++w.phase;
        ++g_clock;
    } else {
        while (*const_cast<volatile uint32_t*>(&w.phase) == phase) yield();
    }
    return w.value[phase & 1u];
}

struct Index {
    uint32_t x;
};

template <class T>
T checked(const T* p)
{
    const char* c = reinterpret_cast<const char*>(p);
    for (const Tables& t : g_tables) {
        const char* const* range = sizeof(T) == 16 ? t.quads : sizeof(T) == 2 ? t.entries : t.all;
        if (c >= range[0] && c + sizeof(T) <= range[1]) return *p;
    }
    std::printf("read of %zu bytes outside its table\n", sizeof(T));
    std::fflush(stdout);
    std::_Exit(0);
}

}  // namespace

#undef __launch_bounds__
#undef __grid_constant__
#undef __global__
#undef __device__
#undef __host__
#undef __shared__
#define __launch_bounds__(...)
#define __grid_constant__
#define __global__
#define __device__
#define __host__
#define __shared__
#undef __noinline__
#define __noinline__ __attribute__((noinline))
#define threadIdx (Index{g_tid})
#define blockIdx (Index{0u})

template <class T>
T __ldg(const T* p) { return checked(p); }
inline void __syncwarp() { exchange(0); }
inline void __syncthreads()
{
    const uint32_t phase = g_block_phase;
    if (++g_block_arrived == kThreads) {
        g_block_arrived = 0;
        ++g_block_phase;
    } else {
        while (*const_cast<volatile uint32_t*>(&g_block_phase) == phase) yield();
    }
}
inline unsigned __ballot_sync(unsigned, bool v)
{
    const uint64_t* a = exchange(v);
    unsigned r = 0;
    for (int l = 0; l < 32; ++l) r |= static_cast<unsigned>(a[l] != 0) << l;
    return r;
}
inline int __any_sync(unsigned m, bool v) { return __ballot_sync(m, v) != 0; }
template <class T>
T __shfl_sync(unsigned, T v, int from) { return static_cast<T>(exchange(v)[from & 31]); }
template <class T>
unsigned __match_any_sync(unsigned mask, T v)
{
    // the lanes of the mask alone meet here
    Warp& w = g_warps[g_tid / 32];
    const uint32_t phase = w.some_phase;
    w.some[g_tid % 32] = v;
    if (++w.some_arrived == static_cast<uint32_t>(__builtin_popcount(mask))) {
        for (int l = 0; l < 32; ++l) {
            w.peers[l] = 0;
            for (int k = 0; k < 32; ++k) w.peers[l] |= static_cast<unsigned>((mask >> k & 1u) && w.some[k] == w.some[l]) << k;
        }
        w.some_arrived = 0;
        ++w.some_phase;
    } else {
        while (*const_cast<volatile uint32_t*>(&w.some_phase) == phase) yield();
    }
    return w.peers[g_tid % 32];
}
inline int __popc(unsigned v) { return __builtin_popcount(v); }
inline int __ffs(unsigned v) { return __builtin_ffs(static_cast<int>(v)); }
inline int __ffsll(long long v) { return __builtin_ffsll(v); }
inline unsigned __fns(unsigned mask, unsigned, int nth)
{
    for (unsigned l = 0; l < 32; ++l)
        if ((mask >> l & 1u) && --nth == 0) return l;
    return ~0u;
}
template <class T>
T atomicAdd(T* p, T v) { return std::exchange(*p, *p + v); }
template <class T>
T atomicMin(T* p, T v) { return std::exchange(*p, std::min(*p, v)); }
template <class T, class U>
T atomicOr(T* p, U v) { return std::exchange(*p, static_cast<T>(*p | static_cast<T>(v))); }
template <class T, class U>
T atomicExch(T* p, U v) { return std::exchange(*p, static_cast<T>(v)); }
template <class T>
T atomicCAS(T* p, T old, T v) { return *p == old ? std::exchange(*p, v) : *p; }
inline void __nanosleep(unsigned) { yield(); }
inline void __threadfence() {}
// not called: launches run below
extern "C" cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t)
{
    std::abort();
}

// the kernel's one inline assembly statement reads the clock into t
#define asm
#define volatile(...) (t = g_clock)
#include "emp_btc.cu"
#undef volatile
#undef asm

namespace emp {
namespace {
alignas(16) uint32_t g_smem[(227 * 1024) / 4];
}
}  // namespace emp

namespace {

using Kernel = void (*)(emp::BtLaunch);
Kernel g_kernel;
emp::BtLaunch g_launch;

void lane_main()
{
    g_kernel(g_launch);
    g_lanes[g_tid].done = true;
    _longjmp(g_scheduler, 1);
}

void launch(const emp::BtLaunch& P)
{
    g_launch = P;
    for (uint32_t t = 0; t < kThreads; ++t) g_lanes[t].started = g_lanes[t].done = false;
    for (bool any = true; any;) {
        any = false;
        for (volatile uint32_t t = 0; t < kThreads; t = t + 1) {
            Lane& l = g_lanes[t];
            if (l.done) continue;
            any = true;
            g_tid = t;
            if (_setjmp(g_scheduler)) continue;
            if (l.started) _longjmp(l.at, 1);
            l.started = true;
            getcontext(&l.first);
            l.first.uc_stack.ss_sp = l.stack.data();
            l.first.uc_stack.ss_size = l.stack.size();
            l.first.uc_link = nullptr;
            makecontext(&l.first, lane_main, 0);
            setcontext(&l.first);
        }
    }
}

unsigned long long number()
{
    unsigned long long v;
    if (std::scanf("%llu", &v) != 1) std::exit(1);
    return v;
}

}  // namespace

int main()
{
    using namespace emp;
    const bool in_smem = number();
    const uint32_t min_nw = number();
    BtLaunch P;
    BtRunCtl ctl{};
    P.item_budget = number();
    P.out_capacity = number();
    ctl.deadline = number();
    P.stop_at_first = number();
    P.stop_at_any = number();
    const uint32_t puzzles = number();
    std::vector<uint32_t> blob;
    std::vector<uint64_t> offs;  // of the puzzles' blobs
    for (uint32_t i = 0; i < puzzles; ++i) {
        const uint32_t w = number(), h = number();
        std::vector<uint8_t> colours(4 * w * h);
        for (uint8_t& c : colours) c = static_cast<uint8_t>(number());
        PuzzleModel m;
        std::vector<LevelPlan> plan;
        std::string err;
        if (!build_model(w, h, colours.data(), m, err) || !build_plan(m, order_basic(w, h), plan, err)) return 1;
        const std::vector<uint32_t> b = build_compact(m, plan, min_nw);
        if (b.empty() || (i && b[0] != blob[0])) return 1;
        offs.push_back(blob.size());
        blob.insert(blob.end(), b.begin(), b.end());
        P.max_levels = std::max(P.max_levels, m.n);
    }
    std::memcpy(&P.chdr, blob.data(), sizeof(P.chdr));
    P.rec_words = 4 + 128;
    const uint64_t records = number();
    std::vector<uint32_t> rec(records * P.rec_words, 0);
    for (uint64_t i = 0; i < records; ++i) {
        uint32_t* r = &rec[i * P.rec_words];
        r[0] = static_cast<uint32_t>(i);
        r[3] = static_cast<uint32_t>(number());
        r[2] = static_cast<uint32_t>(number());
        for (uint32_t j = 0; j < r[2]; ++j) r[4 + (j >> 1)] |= static_cast<uint32_t>(number()) << (16 * (j & 1));
    }
    if (in_smem && puzzles != 1) return 1;
    P.smem_tab_words = in_smem ? P.chdr.hot : 0;
    if (4 * (P.smem_tab_words + kThreads * compact_stack_levels(P.max_levels)) > sizeof(g_smem)) return 1;
    P.ctables = blob.data();
    P.coffset = offs.data();
    for (uint64_t o : offs) {
        CompactHeader h;
        std::memcpy(&h, &blob[o], sizeof(h));
        auto at = [&](uint32_t word) { return reinterpret_cast<const char*>(blob.data() + o + word); };
        // (staging copies the hot part, header included, 16 bytes at a time)
        g_tables.push_back({{at(in_smem ? 0 : h.desc), at(in_smem ? h.hot : h.entries)},
                            {at(h.entries), at(h.hot)},
                            {at(0), at(h.words)}});
    }
    P.crec_words = compact_state_words(P.max_levels, P.chdr.nw);
    P.items_off = static_cast<uint64_t>(P.crec_words) * kThreads;
    P.stack_levels = compact_stack_levels(P.max_levels);
    // 64-bit storage: states hold 64-bit words, and items follow them
    std::vector<unsigned long long> queue[2];
    for (auto& q : queue) q.resize((P.items_off + 1) / 2 + P.out_capacity + 4, 0);
    unsigned long long counters[2];
    std::vector<unsigned long long> totals(2 * puzzles, 0), first_item(puzzles, ~0ull);
    std::vector<FirstRecord> first(puzzles);
    std::memset(first.data(), 0, sizeof(FirstRecord) * puzzles);
    std::vector<uint32_t> incomplete(puzzles, 0);
    int abort_flag = 0, status = 0;
    P.cursor = counters;
    P.out_tail = counters + 1;
    P.totals = totals.data();
    P.first_item = first_item.data();
    P.first_records = first.data();
    P.incomplete = incomplete.data();
    P.abort_flag = &abort_flag;
    P.status = &status;
    P.ctl = &ctl;
    g_kernel = reinterpret_cast<Kernel>(
        const_cast<void*>(compact_kernel_symbol(P.chdr.nw, in_smem, false, kThreads)));
    P.in_rec = rec.data();
    P.n_in = records;
    uint32_t rounds = 0, full = 0;
    while (P.n_in) {
        counters[0] = counters[1] = 0;
        P.out_rec = reinterpret_cast<uint32_t*>(queue[rounds & 1].data());
        P.in_items = rounds != 0;
        launch(P);
        full += counters[1] > P.out_capacity;
        P.n_in = std::min<unsigned long long>(counters[1], P.out_capacity);
        P.in_rec = P.out_rec;
        ++rounds;
    }
    for (uint32_t i = 0; i < puzzles; ++i)
        std::printf("%llu %llu %u\n", totals[2 * i], totals[2 * i + 1], incomplete[i]);
    std::printf("end %llu rounds %u full %u\n", g_clock, rounds, full);
    return 0;
}
