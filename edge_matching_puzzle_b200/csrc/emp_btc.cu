// Exhaustive backtracker over the compact search tables (emp_compact.h): the default search
// of row-major orders.
//
// The search and its initial records are those of dfs_kernel (emp_bt.cu); what differs is what a
// placement costs.  A level's candidates are one row of the tables and the availability, one
// AND of 64 bits for boards of up to about 62 centre pieces, where dfs_kernel combines three
// 64-bit words of piece x orientation bits, searches them and keeps a set apart for identical
// pieces.  Availability stays in registers, and a step looks one level ahead: it takes the
// next candidate of the level, counts it, and goes down only when that leaves the next level
// a candidate, so a dead end costs no stack traffic and no step back.
//
// A step of a warp runs (1) a pop for the lanes whose level is exhausted, (2) the next candidate
// for all lanes that have one, (3) the way down for those whose candidate allows it.  A lane
// whose pop found nothing left there pops again at the next step.  What is rare (flagged rows,
// solutions) is left to a vote of the warp, so the common path has two divergent regions.  The set
// left at a level is not stored: a pop recomputes it as the row AND the availability (which is the
// level's entry availability again) above the slot placed there, with the trials of flagged rows
// replayed (emp_compact.h).
//
// The stack keeps one 32-bit word a level:
//   south colour | slot << 8 | more << 16 | space << 17 | (byte offset of the row / 16) << 18
// (more: candidates remained after this one was taken).  A is the availability of the space
// of the current level and O the other one; they change places when the level's space does.
//
// What bounds it: integer instructions (ALU pipe 78.5 % and issue slots 76.8 % busy in the main
// rounds on a B200, 21 lanes in an instruction, 20 warps an SM, which hide the shared-memory
// latency); 30 of 32 lanes have work at a step, 22 of them a candidate.  Measured, 1/64 of the
// 8x8 tree of 4 border / 8 interior colours, seed 0 (2.77e9 placements): 62.9 ms with dfs_kernel
// (4.4e10 placements/s), 23.3 ms here (1.19e11/s).
// 128-thread blocks, five an SM, let a thread have its 90 registers: 20 warps at 23.4 ms, where 24 warps
// of 80 registers (256-thread blocks) take 24.2 ms and 16 of 128 registers 24.0 ms; on
// 1/1024 of the tree 3.07 against 3.4 ms.  Tried and slower: selects in place of the step's two
// divergent regions (10 %), a second pop in a step (5 %).
#include "emp_bt.h"

#include <cuda_runtime.h>

#include <algorithm>

namespace emp {

namespace {

constexpr unsigned kFull = 0xFFFFFFFFu;

// Work handed from one round to the next: a thread writes its whole state once, and one item
// per level of it that still holds candidates.  A state, 32-bit words: [0,1] subtree, [2] level
// L, [3] puzzle, [4] row of L, [5] first slot left at L, [6,7] border availability, then the
// centre availability (nw 64-bit words) and the stack words of levels 0..L-1.  An item, 64
// bits: state << 32 | level (kNoItem: none).
constexpr unsigned long long kNoItem = ~0ull;
constexpr uint32_t kEmptyRec = 1u << 17;  // initial records: nothing to search
__host__ __device__ constexpr uint32_t state_header(uint32_t nw) { return (8 + 2 * nw + 3) & ~3u; }

__device__ __forceinline__ uint64_t global_ns()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

extern __shared__ __align__(16) uint32_t g_smem[];

__device__ __forceinline__ uint64_t ldg64(const uint32_t* p)
{
    return __ldg(reinterpret_cast<const unsigned long long*>(p));
}

template <int NW>
struct Search {
    uint64_t orig, nodes;
    const uint32_t* tb;              // the puzzle's blob, number and levels: read by plans of several
    uint32_t pz, n;                  // puzzles alone (blob, puzzle and levels below)
    uint32_t L, base, space;
    int row;                         // byte offset of level L's row
    int entries;                     // byte offset of its slot 0 entry
    uint64_t R[NW];                  // candidates left at level L
    uint64_t A[NW], O[NW];           // availability of level L's space, of the other space
    bool active;
};

template <int NW>
struct Row {
    uint64_t m[NW];
    int entries;
    uint32_t clears;
};

// With staged tables the plan has one puzzle: its blob comes first and the rest is in the launch
// parameters, which keeps six registers out of the search.
template <bool SM, int NW>
__device__ __forceinline__ const uint32_t* blob(const BtLaunch& P, const Search<NW>& s)
{
    return SM ? P.ctables : s.tb;
}
template <bool SM, int NW>
__device__ __forceinline__ uint32_t puzzle(const Search<NW>& s)
{
    return SM ? 0u : s.pz;
}
template <bool SM, int NW>
__device__ __forceinline__ uint32_t levels(const BtLaunch& P, const Search<NW>& s)
{
    return SM ? P.chdr.n : s.n;
}

struct SlotBits {
    uint64_t toggle, above;
};

// Table access by byte offset from the blob's start: SM = the plan's single puzzle, hot tables
// staged in shared memory; otherwise read through the read-only path.
template <bool SM, int NW>
struct Tab {
    using S = Search<NW>;
    static __device__ __forceinline__ uint4 quad(const S& s, int off)
    {
        return SM ? *reinterpret_cast<const uint4*>(reinterpret_cast<const char*>(g_smem) + off)
                  : __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const char*>(s.tb) + off));
    }
    static __device__ __forceinline__ uint4 desc(const S& s, uint32_t l) { return quad(s, 4 * kCompactHeader + 16 * l); }
    static __device__ __forceinline__ SlotBits slot(const BtLaunch& P, const S& s, uint32_t space, uint32_t slot)
    {
        const uint32_t at = SM ? 4 * P.chdr.slots : 4 * kCompactHeader + 16 * (s.n + 1);
        const uint4 v = quad(s, at + 16 * (space * (64 * NW) + slot));
        return {v.x | static_cast<uint64_t>(v.y) << 32, v.z | static_cast<uint64_t>(v.w) << 32};
    }
    static __device__ __forceinline__ Row<NW> row(const S& s, int off)
    {
        Row<NW> r;
        const uint4 v = quad(s, off);
        r.m[0] = v.x | static_cast<uint64_t>(v.y) << 32;
        if (NW == 1) {
            r.entries = v.z;
            r.clears = v.w;
        } else {
            r.m[NW > 1] = v.z | static_cast<uint64_t>(v.w) << 32;
            uint4 u = quad(s, off + 16);
            if (NW > 2) {
                r.m[NW > 2 ? 2 : 0] = u.x | static_cast<uint64_t>(u.y) << 32;
                r.m[NW > 2 ? 3 : 0] = u.z | static_cast<uint64_t>(u.w) << 32;
                u = quad(s, off + 32);
            }
            r.entries = u.x;
            r.clears = u.y;
        }
        return r;
    }
    static __device__ __forceinline__ uint32_t entry(const S& s, int entries, uint32_t slot)
    {
        const int off = entries + 2 * static_cast<int>(slot);
        return SM ? *reinterpret_cast<const uint16_t*>(reinterpret_cast<const char*>(g_smem) + off)
                  : __ldg(reinterpret_cast<const uint16_t*>(reinterpret_cast<const char*>(s.tb) + off));
    }
};

__device__ __forceinline__ uint32_t word_slot(uint32_t w) { return (w >> 8) & 0xFFu; }
__device__ __forceinline__ bool word_more(uint32_t w) { return (w >> 16) & 1u; }
__device__ __forceinline__ uint32_t word_space(uint32_t w) { return (w >> 17) & 1u; }
__device__ __forceinline__ int word_row(uint32_t w) { return static_cast<int>((w >> 14) & 0x3FFF0u); }
__device__ __forceinline__ uint32_t make_word(uint32_t e, uint32_t slot, bool more, uint32_t space, int row)
{
    return (e >> 9) | (slot << 8) | (static_cast<uint32_t>(more) << 16) | (space << 17) |
           (static_cast<uint32_t>(row) << 14);
}
// byte offset of the row at a level with descriptor d: west entry and north colour
template <int NW>
__device__ __forceinline__ int row_at(uint4 d, uint32_t west, uint32_t north)
{
    return static_cast<int>(d.x) + static_cast<int>((west & d.z & 0x1F0u) * (row_bytes(NW) / 16)) +
           static_cast<int>(north * d.y);
}
__device__ __forceinline__ uint32_t desc_space(uint4 d) { return (d.z >> 16) & 1u; }

template <int NW>
__device__ __forceinline__ bool any(const uint64_t* r)
{
    uint64_t x = r[0];
#pragma unroll
    for (int w = 1; w < NW; ++w) x |= r[w];
    return x != 0;
}

// lowest slot of a set that is not empty
template <int NW>
__device__ __forceinline__ uint32_t first_slot(const uint64_t* r)
{
    uint64_t x = r[NW - 1];
    uint32_t at = 64 * (NW - 1);
#pragma unroll
    for (int w = NW - 2; w >= 0; --w)
        if (r[w]) {
            x = r[w];
            at = 64 * w;
        }
    return at + static_cast<uint32_t>(__ffsll(static_cast<long long>(x))) - 1;
}

// A and O for a level of space `space`
template <int NW>
__device__ __forceinline__ void to_space(Search<NW>& s, uint32_t space)
{
    const bool swap = s.space != space;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
        const uint64_t a = s.A[w], o = s.O[w];
        s.A[w] = swap ? o : a;
        s.O[w] = swap ? a : o;
    }
    s.space = space;
}

// the piece of a slot of the current space: placed or given back
template <int NW>
__device__ __forceinline__ void toggle(uint64_t* a, uint32_t slot, uint64_t bits)
{
#pragma unroll
    for (int w = 0; w < NW; ++w) a[w] ^= NW == 1 || w == static_cast<int>(slot >> 6) ? bits : 0ull;
}

// The candidates of a flagged row that the reference tries: in ascending order, each trial
// taking out what its identical mask removes (emp_position_strategy.h:197-200).
template <int NW>
struct Set {
    uint64_t w[NW];
};

template <int NW>
__device__ __forceinline__ Set<NW> replay_trials(const uint32_t* id, Set<NW> left)
{
    Set<NW> r{};
    while (any<NW>(left.w)) {
        const uint32_t slot = first_slot<NW>(left.w);
#pragma unroll
        for (int w = 0; w < NW; ++w) {
            const uint64_t bit = w == static_cast<int>(slot >> 6) ? 1ull << (slot & 63u) : 0ull;
            r.w[w] |= bit;
            left.w[w] &= ~(bit | ldg64(id + 2 * (slot * NW + w)));
        }
    }
    return r;
}

// leaves the candidates that are tried in `r`, the candidates of a flagged row
template <int NW>
__device__ __forceinline__ void only_tried(const uint32_t* id, uint64_t* r)
{
    if (NW == 1 && !(r[0] & (r[0] - 1))) return;
    Set<NW> v;
#pragma unroll
    for (int w = 0; w < NW; ++w) v.w[w] = r[w];
    v = replay_trials<NW>(id, v);
#pragma unroll
    for (int w = 0; w < NW; ++w) r[w] = v.w[w];
}

// the current level's candidates: its row AND the availability, without those that other trials
// of a flagged row remove
template <bool SM, int NW>
__device__ __forceinline__ void level_candidates(const BtLaunch& P, Search<NW>& s)
{
    const Row<NW> r = Tab<SM, NW>::row(s, s.row);
    s.entries = r.entries;
#pragma unroll
    for (int w = 0; w < NW; ++w) s.R[w] = r.m[w] & s.A[w];
    if (static_cast<int64_t>(r.m[NW - 1]) < 0) only_tried<NW>(blob<SM>(P, s) + r.clears, s.R);
}

// whether a row's trials have to be replayed
template <int NW>
__device__ __forceinline__ bool flagged(const Row<NW>& row)
{
    return static_cast<int64_t>(row.m[NW - 1]) < 0;
}

// of those, the ones above a slot
template <int NW>
__device__ __forceinline__ void above_slot(uint64_t* r, uint32_t slot, uint64_t above)
{
    if (NW == 1) {
        r[0] &= above;
    } else {
#pragma unroll
        for (int w = 0; w < NW; ++w)
            r[w] = w < static_cast<int>(slot >> 6) ? 0ull : (w == static_cast<int>(slot >> 6) ? r[w] & above : r[w]);
    }
}

// transition (kind_index << 2 | orientation) of a stack word
template <bool SM, int NW>
__device__ __forceinline__ uint32_t word_transition(const BtLaunch& P, const Search<NW>& s, uint32_t word)
{
    const uint32_t slot = word_slot(word), space = word_space(word);
    const uint32_t* tb = blob<SM>(P, s);
    uint32_t ki = __ldg(reinterpret_cast<const uint8_t*>(tb + __ldg(tb + 9)) + space * 64 * NW + slot);
    const uint32_t nborder = __ldg(tb + 11);
    if (space && ki >= nborder) ki -= nborder;
    return (ki << 2) | (Tab<SM, NW>::entry(s, Tab<SM, NW>::row(s, word_row(word)).entries, slot) & 3u);
}

// (The functions below that are not inlined take the state by value: a reference would keep
// the state of the whole kernel in local memory.)

template <bool SM, int NW>
__device__ __forceinline__ void start_puzzle(const BtLaunch& P, Search<NW>& s, uint32_t pz)
{
    s.pz = pz;
    s.tb = P.ctables + P.coffset[pz];
    s.n = SM ? P.chdr.n : __ldg(s.tb + 1);
    s.space = 0;
}

template <int NW>
__device__ __forceinline__ void start_search(Search<NW>& s, uint32_t len)
{
    s.L = len;
    s.base = len;
    s.nodes = 0;
    s.active = true;
}

// no work: an empty set at the base level
template <int NW>
__device__ __forceinline__ void idle(Search<NW>& s)
{
    s.active = false;
    s.L = 0;
    s.base = 0;
    s.nodes = 0;
#pragma unroll
    for (int w = 0; w < NW; ++w) s.R[w] = 0;
}

// Starts an item of an earlier round: level `len` of a handed-back state, after the piece
// placed there (or from the state's first slot when it is the state's own level).
template <bool SM, int NW, int T>
__device__ __forceinline__ void load_item(const BtLaunch& P, Search<NW>& s, const uint32_t* st, uint32_t len,
                                          uint32_t* stk)
{
    const uint4 h = *reinterpret_cast<const uint4*>(st), g = *reinterpret_cast<const uint4*>(st + 4);
    s.orig = static_cast<uint64_t>(h.x) | (static_cast<uint64_t>(h.y) << 32);
    start_puzzle<SM, NW>(P, s, h.w);
#pragma unroll
    for (int w = 0; w < NW; ++w) {
        s.A[w] = *reinterpret_cast<const uint64_t*>(st + 8 + 2 * w);
        s.O[w] = w ? 0ull : g.z | static_cast<uint64_t>(g.w) << 32;
    }
    s.row = static_cast<int>(g.x);
    // the whole stack first, four loads of four words on their way at a time ...
    const uint4* pre = reinterpret_cast<const uint4*>(st + state_header(NW));
    for (uint32_t l = 0; l < h.z; l += 16) {
        uint4 v[4];
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j)
            if (l + 4 * j < h.z) v[j] = pre[l / 4 + j];
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j)
            if (l + 4 * j < h.z) {
                uint32_t* q = stk + (l + 4 * j) * T;
                q[0] = v[j].x;
                q[T] = v[j].y;
                q[2 * T] = v[j].z;
                q[3 * T] = v[j].w;
            }
    }
    // ... then the pieces at and past the level are given back
    for (uint32_t l = len; l < h.z; ++l) {
        const uint32_t word = stk[l * T], slot = word_slot(word);
        to_space<NW>(s, word_space(word));
        toggle<NW>(s.A, slot, Tab<SM, NW>::slot(P, s, word_space(word), slot).toggle);
    }
    to_space<NW>(s, desc_space(Tab<SM, NW>::desc(s, len)));
    if (len < h.z) s.row = word_row(stk[len * T]);
    level_candidates<SM, NW>(P, s);
    // after the piece placed at the level, or from the first slot left at the state's own level
    const uint32_t from = len < h.z ? word_slot(stk[len * T]) + 1 : g.y;
    if (from) above_slot<NW>(s.R, from - 1, Tab<SM, NW>::slot(P, s, s.space, from - 1).above);
    start_search<NW>(s, len);
}

// Starts an initial record: a prefix of transitions from the expansion, or a level of a resumed
// search with the transition it starts from.
template <bool SM, int NW, int T>
__device__ __forceinline__ void load_record(const BtLaunch& P, Search<NW>& s, const uint32_t* rec, uint32_t* stk)
{
    s.orig = static_cast<uint64_t>(rec[0]) | (static_cast<uint64_t>(rec[1]) << 32);
    const uint32_t len = rec[2] & 0xFFFFu, start = rec[2] >> 16;
    start_puzzle<SM, NW>(P, s, rec[3] & 0xFFFFu);
    const uint32_t* tb = blob<SM>(P, s);
    const uint32_t init = __ldg(tb + 8), nborder = __ldg(tb + 11);
    const uint32_t width = SM ? P.chdr.width : __ldg(tb + 2);
    const uint8_t* first = reinterpret_cast<const uint8_t*>(tb + __ldg(tb + 10));
#pragma unroll
    for (int w = 0; w < NW; ++w) {
        s.A[w] = ldg64(tb + init + 2 + 2 * w);
        s.O[w] = w ? 0ull : ldg64(tb + init);
    }
    uint32_t west = 0;
    for (uint32_t l = 0;; ++l) {
        const uint4 d = Tab<SM, NW>::desc(s, l);
        const uint32_t north = l ? stk[d.w * T] & 0xFFu : 0u;
        s.row = row_at<NW>(d, west, north);
        to_space<NW>(s, desc_space(d));
        if (l == len) break;
        const uint32_t t = (rec[4 + (l >> 1)] >> (16 * (l & 1))) & 0xFFFFu;
        // corners follow the borders in space 1
        const bool corner = l == 0 || l + 1 == width || l + width == levels<SM>(P, s) || l + 1 == levels<SM>(P, s);
        uint32_t slot = __ldg(first + 256 * s.space + (t >> 2) + (corner ? nborder : 0u));
        const int entries = Tab<SM, NW>::row(s, s.row).entries;
        uint32_t e = Tab<SM, NW>::entry(s, entries, slot);
        // the piece's slots in this row ascend with the orientation
        for (int k = 0; k < 3 && (e & 3u) != (t & 3u); ++k) e = Tab<SM, NW>::entry(s, entries, ++slot);
        toggle<NW>(s.A, slot, Tab<SM, NW>::slot(P, s, s.space, slot).toggle);
        stk[l * T] = make_word(e, slot, false, s.space, s.row);
        west = e;
    }
    level_candidates<SM, NW>(P, s);
    if (start) {
        // a resumed level: drop the candidates below transition `start`
        while (any<NW>(s.R)) {
            const uint32_t slot = first_slot<NW>(s.R);
            if (word_transition<SM, NW>(P, s, make_word(0, slot, false, s.space, s.row)) >= start) break;
#pragma unroll
            for (int w = 0; w < NW; ++w)
                if (w == static_cast<int>(slot >> 6)) s.R[w] &= s.R[w] - 1;
        }
    }
    start_search<NW>(s, len);
}

// whether this solution's path comes before the recorded one
template <bool SM, int NW, int T>
__device__ __forceinline__ bool path_before(const BtLaunch& P, const Search<NW>& s, const uint32_t* stk,
                                            const FirstRecord* r)
{
    for (uint32_t l = 0; l < levels<SM>(P, s); ++l) {
        const uint32_t mine = word_transition<SM, NW>(P, s, stk[l * T]);
        const uint32_t theirs = *reinterpret_cast<const volatile uint16_t*>(&r->t[l]);
        if (mine != theirs) return mine < theirs;
    }
    return false;
}

// Keeps the lexicographically smallest solution path of each puzzle, as record_solution of
// emp_bt.cu does (bounded wait for the record's lock).  The record only ever improves, so a path
// that does not come before an unchanged copy of it needs no lock: `version` is odd while the
// record is written.  Lanes that share the lowest subtree find its solutions at once, and on boards
// with millions of them all waited for the lock: 7x7 of 1/2 colours, split at level 6, counted 4e8
// placements/s and ended 0.56 s after a deadline of 0.2 s; now 4.4e10 and 7 ms.
template <bool SM, int NW, int T>
__device__ __forceinline__ void record_solution(const BtLaunch& P, const Search<NW>& s, const uint32_t* stk)
{
    FirstRecord* r = P.first_records + puzzle<SM>(s);
    // (the lowest subtree only falls: mostly a look is enough)
    const unsigned long long lowest = *(volatile unsigned long long*)&P.first_item[puzzle<SM>(s)];
    if (s.orig > lowest) return;
    if (s.orig < lowest && atomicMin(&P.first_item[puzzle<SM>(s)], (unsigned long long)s.orig) < s.orig) return;
    const uint32_t version = *(volatile unsigned int*)&r->version;
    if (version && !(version & 1u)) {
        __threadfence();
        const bool before = path_before<SM, NW, T>(P, s, stk, r);
        __threadfence();
        if (!before && *(volatile unsigned int*)&r->version == version) return;
    }
    const uint64_t give_up = global_ns() + P.first_lock_wait_ns;
    while (atomicCAS(&r->lock, 0u, 1u) != 0u) {
        if (global_ns() > give_up) {
            atomicExch(&r->missed, 1u);
            atomicOr(P.status, EMP_DEV_FIRST_LOST);
            return;
        }
        __nanosleep(64);
    }
    __threadfence();
    if (!r->has || path_before<SM, NW, T>(P, s, stk, r)) {
        atomicAdd(&r->version, 1u);
        __threadfence();
        for (uint32_t l = 0; l < levels<SM>(P, s); ++l)
            r->t[l] = static_cast<uint16_t>(word_transition<SM, NW>(P, s, stk[l * T]));
        r->has = 1;
        __threadfence();
        atomicAdd(&r->version, 1u);
    }
    __threadfence();
    atomicExch(&r->lock, 0u);
}

// A solution's whole path is on the stack (its last piece's word included).  who: the lanes of the
// warp that found one at this step.  They are counted together, for an addition each to one address
// and one to the lowest subtree took 40 % of a search in which 1.2 % of the placements are solutions
// (8x8 of 1/3 colours: 3.0e10 placements/s so, 5.0e10 now).
template <bool SM, int NW, int T>
__device__ __noinline__ void solution_found(const BtLaunch& P, const Search<NW> s, const uint32_t* stk,
                                            uint32_t placed, unsigned who)
{
    const unsigned peers = SM ? who : __match_any_sync(who, s.pz);
    if ((threadIdx.x & 31u) == __ffs(peers) - 1)
        atomicAdd(&P.totals[2 * puzzle<SM>(s) + 1], static_cast<unsigned long long>(__popc(peers)));
    if (P.item_nodes) atomicAdd(&P.item_sols[s.orig], 1ull);
    record_solution<SM, NW, T>(P, s, stk);
    if (P.sols) {
        const unsigned long long at = atomicAdd(P.sol_count, 1ull);
        if (at < P.sol_capacity) {
            SolutionRecord* r = P.sols + at;
            r->orig = s.orig;
            r->local = s.nodes + placed;
            for (uint32_t l = 0; l < levels<SM>(P, s); ++l)
                r->t[l] = static_cast<uint16_t>(word_transition<SM, NW>(P, s, stk[l * T]));
        }
    }
    if (P.stop_at_any) {
        // first solution of the run: note the time and stop every thread
        atomicCAS(&P.ctl->first_found_ns, 0ull, static_cast<unsigned long long>(global_ns()));
        atomicExch(P.abort_flag, 1);
    }
}

template <bool SM, int NW>
__device__ __forceinline__ void account(const BtLaunch& P, const Search<NW>& s)
{
    if (s.nodes) atomicAdd(&P.totals[2 * puzzle<SM>(s)], (unsigned long long)s.nodes);
    if (P.item_nodes) {
        if (s.nodes) atomicAdd(&P.item_nodes[s.orig], (unsigned long long)s.nodes);
    }
}

// Hands the remaining work of the thread to the next round: its state, in the slot that is this
// thread's own, and one item per level that still holds candidates (the more bits say which).
// Returns false when the item queue is full (the thread then keeps the work; the plans' queues hold
// every open level, so theirs never fill).  A state slot is written once a round, since items point
// to it: a lane that handed back may take work again from a neighbour that could not
// (share_in_warp), but its own next attempt fails too, for the queue's tail never falls, and once a
// neighbour did not fit nothing fits.  A rule that hands back at another time has to keep that.
template <bool SM, int NW, int T>
__device__ __noinline__ bool split_state(const BtLaunch& P, uint32_t* out, const Search<NW> s, const uint32_t* stk)
{
    const bool here = any<NW>(s.R);
    uint32_t cnt = here;
    for (uint32_t l = s.base; l < s.L; ++l) cnt += word_more(stk[l * T]);
    if (!cnt) return true;
    unsigned long long* items = reinterpret_cast<unsigned long long*>(out + P.items_off);
    unsigned long long k = atomicAdd(P.out_tail, (unsigned long long)cnt);
    if (k + cnt > P.out_capacity) {
        for (; cnt && k < P.out_capacity; ++k, --cnt) items[k] = kNoItem;  // reserved places that fit
        return false;
    }
    const unsigned long long me = blockIdx.x * T + threadIdx.x;
    for (uint32_t l = s.base; l < s.L; ++l)
        if (word_more(stk[l * T])) items[k++] = (me << 32) | l;
    if (here) items[k] = (me << 32) | s.L;
    uint32_t* st = out + me * P.crec_words;
    *reinterpret_cast<uint4*>(st) =
        make_uint4(static_cast<uint32_t>(s.orig), static_cast<uint32_t>(s.orig >> 32), s.L, puzzle<SM>(s));
    const uint64_t border = s.space ? s.A[0] : s.O[0];
    *reinterpret_cast<uint4*>(st + 4) = make_uint4(static_cast<uint32_t>(s.row), here ? first_slot<NW>(s.R) : 0u,
                                                   static_cast<uint32_t>(border), static_cast<uint32_t>(border >> 32));
#pragma unroll
    for (int w = 0; w < NW; ++w) *reinterpret_cast<uint64_t*>(st + 8 + 2 * w) = s.space ? s.O[w] : s.A[w];
    uint32_t* pre = st + state_header(NW);
    for (uint32_t l = 0; l < s.L; l += 4)  // the stack column holds a multiple of 4 levels
        *reinterpret_cast<uint4*>(pre + l) =
            make_uint4(stk[l * T], stk[(l + 1) * T], stk[(l + 2) * T], stk[(l + 3) * T]);
    return true;
}

// Once a round's queue is empty, idle lanes of a warp take work from its busy ones: the rest of
// their shallowest open level.  The thief copies the path down to that level and gives back, in
// its copy of the availability, the pieces from there on; the donor, all of whose shallower
// levels are exhausted, ends its search above that level.  Measured on a B200 (split budget 64
// without sharing, 256 with it): a 7x7 count of 2.3e6 placements 0.56 ms in 13 rounds -> 0.37 ms
// in 5; 1/1024 of the tree above 3.84 -> 3.43 ms, 1/64 25.3 -> 25.7 ms at the same 30 -> 16 rounds.
// A lane whose subtree a lower solution supersedes gives nothing away: the two would pass the work
// to and fro, each for the 4096 steps between its looks at the flags.
template <bool SM, int NW, int T>
__device__ __noinline__ Search<NW> share_in_warp(const BtLaunch& P, Search<NW> s, uint32_t* stk)
{
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t open = ~0u;
    const bool wanted =
        !(P.stop_at_first && s.active && s.orig > *(volatile unsigned long long*)&P.first_item[puzzle<SM>(s)]);
    if (s.active && wanted)
        for (uint32_t l = s.base; l < s.L; ++l)
            if (word_more(stk[l * T])) {
                open = l;
                break;
            }
    __syncwarp();
    const unsigned donors = __ballot_sync(kFull, open != ~0u), idle = __ballot_sync(kFull, !s.active);
    if (!donors) return s;
    const uint32_t lt = (1u << lane) - 1u;
    const bool thief = !s.active && __popc(idle & lt) < __popc(donors);
    const bool donor = open != ~0u && __popc(donors & lt) < __popc(idle);
    const uint32_t from = thief ? __fns(donors, 0, __popc(idle & lt) + 1) : lane;
    const uint32_t level = __shfl_sync(kFull, open, from), top = __shfl_sync(kFull, s.L, from);
    const uint32_t space = __shfl_sync(kFull, s.space, from), pz = __shfl_sync(kFull, puzzle<SM>(s), from);
    const uint64_t orig = __shfl_sync(kFull, s.orig, from);
    uint64_t a[NW], o[NW];
#pragma unroll
    for (int w = 0; w < NW; ++w) {
        a[w] = __shfl_sync(kFull, s.A[w], from);
        o[w] = __shfl_sync(kFull, s.O[w], from);
    }
    if (thief) {
        const uint32_t* col = stk + static_cast<int>(from) - static_cast<int>(lane);
        s.orig = orig;
        start_puzzle<SM, NW>(P, s, pz);
        s.space = space;
#pragma unroll
        for (int w = 0; w < NW; ++w) {
            s.A[w] = a[w];
            s.O[w] = o[w];
        }
#pragma unroll 4
        for (uint32_t l = 0; l < level; ++l) stk[l * T] = col[l * T];
        for (uint32_t l = level; l < top; ++l) {
            const uint32_t word = col[l * T], slot = word_slot(word);
            to_space<NW>(s, word_space(word));
            toggle<NW>(s.A, slot, Tab<SM, NW>::slot(P, s, word_space(word), slot).toggle);
        }
        const uint32_t word = col[level * T], slot = word_slot(word);
        to_space<NW>(s, word_space(word));
        s.row = word_row(word);
        level_candidates<SM, NW>(P, s);
        above_slot<NW>(s.R, slot, Tab<SM, NW>::slot(P, s, s.space, slot).above);
        start_search<NW>(s, level);
    }
    __syncwarp();
    if (donor) {
        stk[open * T] &= ~(1u << 16);
        s.base = open + 1;
    }
    __syncwarp();
    return s;
}

// Persistent search over the records of a round; the fetch and the checks of the deadline,
// cancellation and stop-at-first flags are those of dfs_kernel.  Work goes back to the queue for
// the next round once a warp has searched on for the split budget after the queue ran empty.
template <int NW, bool SM, bool GS, int T, int kStepsPerFetch>
__global__ void __launch_bounds__(T, (NW == 1 && SM ? (T == 128 ? 640 : 768) : 512) / T)
    dfs_compact_kernel(const __grid_constant__ BtLaunch P)
{
    using TB = Tab<SM, NW>;
    const uint32_t tid = threadIdx.x, lane = tid & 31;
    if (SM) {
        const uint4* src = reinterpret_cast<const uint4*>(P.ctables + P.coffset[0]);
        uint4* dst = reinterpret_cast<uint4*>(g_smem);
        for (uint32_t i = tid; i < P.smem_tab_words / 4; i += T) dst[i] = __ldg(src + i);
        __syncthreads();
    }
    uint32_t* const stk = GS ? P.stack + (size_t)blockIdx.x * T * P.stack_levels + tid : g_smem + P.smem_tab_words + tid;
    Search<NW> s;
    idle<NW>(s);
    bool fix = false;          // the level's candidates still hold what its row's trials remove
    bool alive = true;
    bool stopped = false;      // this lane saw the run's deadline or abort flag
    bool drained = false;      // warp-uniform: the input queue of this round is empty
    uint32_t iteration = 0;    // warp-uniform loop counter
    uint32_t alone = 0;        // warp-uniform: steps since the warp found the queue empty (no more
                               // than it takes to compare)
    uint32_t since_check = 0;  // steps since the last look at the global flags
    const uint64_t deadline = *(volatile unsigned long long*)&P.ctl->deadline;
    const uint64_t n_in = P.n_in_from_ctl ? *(volatile unsigned long long*)&P.ctl->n_in : P.n_in;
    // rounds after the first read what the one before handed back; in graph runs the two
    // queues change roles every round
    const uint32_t* in = P.in_rec;
    uint32_t* out = P.out_rec;
    if (P.swap_rec) {
        if (*(volatile unsigned long long*)&P.ctl->rounds & 1ull) {
            in = P.out_rec;
            out = P.swap_rec;
        } else {
            in = P.swap_rec;
        }
    }
    const unsigned long long* items =
        P.in_items ? reinterpret_cast<const unsigned long long*>(in + P.items_off) : nullptr;
    const uint32_t lt_mask = (1u << lane) - 1u;

    for (;; ++iteration) {
        // ---- work fetch: one atomic per warp, ranks from the ballot ----
        // a lane that dropped its work (handed back, stopped, superseded) may have just entered a
        // flagged row: what it takes next starts from sets whose trials are replayed already
        if (!s.active) fix = false;
        if (drained && !s.active) alive = false;
        const bool need = alive && !s.active;
        const unsigned needmask = __ballot_sync(kFull, need);
        if (needmask) {
            const uint32_t leader = __ffs(needmask) - 1;
            unsigned long long base = 0;
            if (lane == leader) base = atomicAdd(P.cursor, (unsigned long long)__popc(needmask));
            base = __shfl_sync(kFull, base, leader);
            if (base + __popc(needmask) >= n_in) drained = true;
            if (need) {
                const uint64_t my = base + __popc(needmask & lt_mask);
                if (my < n_in) {
                    const unsigned long long item = items ? items[my] : 0ull;
                    const uint32_t* rec = in + (items ? (item >> 32) : my) * (items ? P.crec_words : P.rec_words);
                    if (items ? item != kNoItem : !(rec[3] & kEmptyRec)) {
                        if (*(volatile int*)P.abort_flag) {
                            P.incomplete[rec[3] & 0xFFFFu] = 1u;  // stopped: the work stays unsearched
                        } else {
                            if (items) load_item<SM, NW, T>(P, s, rec, static_cast<uint32_t>(item), stk);
                            else load_record<SM, NW, T>(P, s, rec, stk);
                            if (P.stop_at_first && s.orig > *(volatile unsigned long long*)&P.first_item[puzzle<SM>(s)])
                                idle<NW>(s);  // a lower subtree of this puzzle holds a solution
                        }
                    }
                } else {
                    alive = false;
                }
            }
        } else if (!drained && (iteration & 31u) == 31u) {
            // every warp learns within 32 rounds of steps that the queue ran dry
            unsigned long long c = 0;
            if (lane == 0) c = *(volatile unsigned long long*)P.cursor;
            c = __shfl_sync(kFull, c, 0);
            drained = c >= n_in;
        }
        if (drained && P.item_budget) {
            const unsigned busy = __ballot_sync(kFull, s.active);
            // once the run stops, no lane takes on more
            if (busy && busy != kFull && !__any_sync(kFull, stopped)) {
                s = share_in_warp<SM, NW, T>(P, s, stk);
                alive |= s.active;
            }
        }
        if (!__any_sync(kFull, alive)) break;

        // ---- steps: a warp-uniform trip count; a lane without work has an empty set at its
        // base level and sits them out ----
        uint32_t placed = 0;
        for (int step = 0; step < kStepsPerFetch; ++step) {
            // (1) an exhausted level: up to the one before, whose piece is given back
            uint32_t popped = 0;
            if (!any<NW>(s.R) && s.L != s.base) {
                --s.L;
                const uint32_t word = stk[s.L * T], slot = word_slot(word);
                const SlotBits bits = TB::slot(P, s, word_space(word), slot);
                to_space<NW>(s, word_space(word));
                toggle<NW>(s.A, slot, bits.toggle);
                s.row = word_row(word);
                const Row<NW> r = TB::row(s, s.row);
                s.entries = r.entries;
#pragma unroll
                for (int w = 0; w < NW; ++w) s.R[w] = r.m[w] & s.A[w];
                fix = flagged<NW>(r);
                above_slot<NW>(s.R, slot, bits.above);
                popped = slot + 1;
            }
            // the trials of flagged rows, of a level popped to or just entered
            if (__any_sync(kFull, fix)) {
                if (fix) {
                    level_candidates<SM, NW>(P, s);
                    if (popped) above_slot<NW>(s.R, popped - 1, TB::slot(P, s, s.space, popped - 1).above);
                    fix = false;
                }
                __syncwarp();
            }
            // (2) the next candidate of the level, and what it leaves the next one
            bool solved = false;
            if (any<NW>(s.R)) {
                const uint32_t slot = first_slot<NW>(s.R);
#pragma unroll
                for (int w = 0; w < NW; ++w)
                    if (NW == 1 || w == static_cast<int>(slot >> 6)) s.R[w] &= s.R[w] - 1;
                const uint4 d = TB::desc(s, s.L + 1);
                const uint32_t e = TB::entry(s, s.entries, slot);
                const uint64_t bits = TB::slot(P, s, s.space, slot).toggle;
                const uint32_t north = *reinterpret_cast<const uint8_t*>(&stk[d.w * T]);
                const int crow = row_at<NW>(d, e, north);
                const bool same = desc_space(d) == s.space;
                const Row<NW> r = TB::row(s, crow);
                ++placed;
                // this level's word, should the search go down
                stk[s.L * T] = make_word(e, slot, any<NW>(s.R), s.space, s.row);
                uint64_t a[NW], c[NW];
#pragma unroll
                for (int w = 0; w < NW; ++w) {
                    a[w] = s.A[w] ^ (NW == 1 || w == static_cast<int>(slot >> 6) ? bits : 0ull);
                    c[w] = r.m[w] & (same ? a[w] : s.O[w]);
                }
                solved = s.L == levels<SM>(P, s) - 1;  // level n has no candidate
                // (3) down, when the next level has one
                if (any<NW>(c)) {
                    fix = flagged<NW>(r);
#pragma unroll
                    for (int w = 0; w < NW; ++w) {
                        const uint64_t o = s.O[w];
                        s.A[w] = same ? a[w] : o;
                        s.O[w] = same ? o : a[w];
                        s.R[w] = c[w];
                    }
                    s.space = same ? s.space : s.space ^ 1u;
                    ++s.L;
                    s.row = crow;
                    s.entries = r.entries;
                }
            }
            if (__any_sync(kFull, solved)) {
                const unsigned who = __ballot_sync(kFull, solved);
                if (solved) {
                    solution_found<SM, NW, T>(P, s, stk, placed, who);
                }
                __syncwarp();
            }
        }
        s.nodes += placed;
        if (s.active && !any<NW>(s.R) && s.L == s.base) {
            account<SM, NW>(P, s);
            idle<NW>(s);
        }
        if (drained && alone < 0x80000000u) alone += kStepsPerFetch;
        if (!s.active) continue;
        since_check += kStepsPerFetch;

        // ---- once the queue is empty, hand work back for the next round ----
        if (P.item_budget && alone >= P.item_budget) {
            if (split_state<SM, NW, T>(P, out, s, stk)) {
                account<SM, NW>(P, s);
                idle<NW>(s);
                alive = false;
                continue;
            }
        }
        // ---- deadline, cancellation and stop-at-first, every 4096 steps ----
        if (since_check >= 4096) {
            since_check = 0;
            bool stop = *(volatile int*)P.abort_flag != 0;
            if (deadline && global_ns() > deadline) {
                stop = true;
                atomicOr(P.status, EMP_DEV_TIMEOUT);
            }
            const bool superseded =
                P.stop_at_first && s.orig > *(volatile unsigned long long*)&P.first_item[puzzle<SM>(s)];
            stopped |= stop;
            if (superseded || stop) {
                account<SM, NW>(P, s);
                if (stop) {
                    // the lane stays alive: it goes on taking records only to mark
                    // their puzzles incomplete, so every dropped piece of work is known
                    P.incomplete[puzzle<SM>(s)] = 1u;
                    atomicExch(P.abort_flag, 1);
                    atomicOr(P.status, EMP_DEV_ABORTED);
                } else {
                    atomicOr(P.status, EMP_DEV_SUPERSEDED);
                }
                idle<NW>(s);
            }
        }
    }
}

// steps between looks at the queue: 16, 32 and 64 took 24.7, 24.2 and 25.1 ms on 1/64 of the
// seed-0 8x8 tree in 256-thread blocks; 32 and 48 took 23.3 and 23.5 ms in 128-thread blocks,
// and 3.17 and 3.07 ms on 1/1024 of it
constexpr int kSteps = 48;

template <int NW, int T>
const void* symbol_t(bool sm, bool gs)
{
    if (sm) return gs ? reinterpret_cast<const void*>(&dfs_compact_kernel<NW, true, true, T, kSteps>)
                      : reinterpret_cast<const void*>(&dfs_compact_kernel<NW, true, false, T, kSteps>);
    return gs ? reinterpret_cast<const void*>(&dfs_compact_kernel<NW, false, true, T, kSteps>)
              : reinterpret_cast<const void*>(&dfs_compact_kernel<NW, false, false, T, kSteps>);
}

template <int T>
const void* symbol_nw(uint32_t nw, bool sm, bool gs)
{
    switch (nw) {
        case 1: return symbol_t<1, T>(sm, gs);
        case 2: return symbol_t<2, T>(sm, gs);
        case 4: return symbol_t<4, T>(sm, gs);
        default: return nullptr;
    }
}

}  // namespace

const void* compact_kernel_symbol(uint32_t nw, bool smem_tables, bool global_stack, uint32_t threads)
{
    switch (threads) {
        case 128: return symbol_nw<128>(nw, smem_tables, global_stack);
        case 256: return symbol_nw<256>(nw, smem_tables, global_stack);
        case 512: return symbol_nw<512>(nw, smem_tables, global_stack);
        default: return nullptr;
    }
}

uint32_t compact_state_words(uint32_t max_levels, uint32_t nw)
{
    return state_header(nw) + compact_stack_levels(max_levels);
}

uint32_t compact_stack_levels(uint32_t max_levels) { return (max_levels + 3) & ~3u; }

size_t compact_smem_bytes(uint32_t max_levels, uint32_t threads, uint32_t tab_words, bool global_stack)
{
    return sizeof(uint32_t) * (static_cast<size_t>(tab_words) +
                               (global_stack ? 0 : static_cast<size_t>(compact_stack_levels(max_levels)) * threads));
}

cudaError_t launch_dfs_compact(const BtLaunch& P, uint32_t blocks, uint32_t threads, cudaStream_t stream)
{
    const bool gs = P.stack != nullptr;
    const void* fn = compact_kernel_symbol(P.chdr.nw, P.smem_tab_words != 0, gs, threads);
    if (!fn) return cudaErrorInvalidValue;
    const size_t smem = compact_smem_bytes(P.max_levels, threads, P.smem_tab_words, gs);
    void* args[] = {const_cast<BtLaunch*>(&P)};
    return cudaLaunchKernel(fn, dim3(blocks), dim3(threads), args, smem, stream);
}

}  // namespace emp
