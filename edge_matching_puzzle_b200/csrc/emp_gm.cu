// Glutton max search for sm_100a.
//
// The method is the reference's CUDA_glutton_max kernel
// (include/CUDA_glutton_max.h:1522-1637): at every level
//   1. remove_invalid_transitions (:745-954): drop every candidate (position,
//      piece, orientation) whose trial placement empties a free position or
//      leaves an available piece with nowhere to go, until nothing changes;
//   2. get_best_candidate (:1010-1301): score every remaining candidate by its
//      trial (total remaining bits over positions and pieces, then
//      (max << 16) + min), keep the first maximum in (info, word, bit) order,
//      the last candidate at the last level;
//   3. apply_best_candidate (:1306-1476): clear its bit, build the next level,
//      push, apply the colour constraints of its sides;
// popping when a level fails (CUDA_glutton_max_stack.h:437-522).
//
// B200 design: 1024-thread blocks keep the level in shared memory together with per-level
// statistics -- orientation counts N[j][q] of piece q at free position j, bit totals A[j],
// per-piece sums S[q] and, per piece, the six smallest and six largest A[j]-N[j][q].  A trial
// then looks at the (at most four) colour-constrained neighbour positions alone; every other
// position contributes A[j]-N[j][p], and the piece counts follow from S[q]-N[i][q] minus what
// the neighbours lost.  This gives the reference's (valid, total, min, max) exactly.  Step 1
// runs as Jacobi passes (all candidates against the same level, then all removals): validity
// only gets harder as bits disappear, so the passes reach the same greatest fixpoint as the
// reference's in-place sweep, and they empty a position exactly when the reference's sweep does.
//
// A trial is made by a group of G lanes, G the words that hold pieces (8, 16 or 32: up to 64,
// 128, 256 pieces), lane w with word w, the pieces 8w..8w+7.  A trial's piece counts are eight
// 16-bit numbers a lane: what position i and its neighbours leave of S (the same for every
// candidate of i, kept in registers) plus what the neighbours keep, counted nibble by nibble
// with bit operations.  The candidates of a pass are dealt out evenly by rank, so a group gets
// a run of neighbouring candidates, nearly all of one position, and no work counter is needed.
//
// What bounds it: the trials' instructions and latency.  Measured on a B200, whole calls:
// 16x16 (5/17 colours, 300 pushes, 148 blocks) 165 ms with a warp per word of candidates and
// full scans for the lists, 42 ms now, 31 us a pass of 43 000 trials; 8x8 on one block (150
// pushes) 162 ms, now 21 ms.
#include "emp_gm.h"

#include <cuda_runtime.h>

namespace emp {

namespace {

constexpr int kThreads = 1024;
constexpr unsigned kFull = 0xFFFFFFFFu;
constexpr uint64_t kBarrierWaitNs = 5000000000ull;  // 5 s: far beyond one validity pass

struct GmSmem {
    alignas(16) uint32_t X[256][32];       // infos of the current level
    uint32_t inval[256][32];   // candidates found invalid in this pass
    alignas(16) uint8_t N[256][256];  // N[j][q]: orientations of piece q left at info j
    uint32_t lo[256][6];       // per piece q: six smallest (A[j]-N[j][q]) << 16 | j, ~0 empty
    uint32_t hi[256][6];       // per piece q: six largest (A[j]-N[j][q]+1) << 16 | j, 0 empty
    uint32_t cc[32][4][32];    // colour constraints
    alignas(16) uint32_t K[256];  // A[j] << 8 | j, ~0 past the last info
    uint32_t cum[257];         // candidates of the infos before j
    uint32_t part[16][64];     // partial sums of N, four pieces a word
    uint16_t A[256];           // bits of info j
    alignas(16) uint16_t S[256];  // sum over j of N[j][q]
    uint16_t rank[4][256];     // partial ranks of K[j]
    uint8_t ord[256];          // infos in ascending order of A
    alignas(4) uint8_t pieces[256][4];
    uint32_t position_index[256];
    uint32_t info_index[256];
    uint32_t played[256];      // this block's copy of the played stack
    uint32_t avail[8];
    unsigned long long warp_key[32];
    uint32_t warp_order[32];
    unsigned long long trials, pushes;  // of the whole search, counted alike by every block
    uint32_t sumA;
    uint32_t any_invalid;
    uint32_t any_empty;
    uint32_t best_order;       // chosen candidate: info << 10 | word << 5 | bit; ~0 none
    uint32_t level, new_level, pop_index, stop, apply_failed;
};

__device__ __forceinline__ uint32_t tri_base(uint32_t S, uint32_t L)
{
    return (S * (S + 1) - (S - L) * (S - L + 1)) / 2;
}

__device__ __forceinline__ uint64_t global_ns()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// get_best_candidate's preference (include/CUDA_glutton_max.h:1196-1295): is candidate
// (k, o) better than (k0, o0)?  order ~0 is "none".  Orders are distinct, so this is a
// strict total order and any reduction tree finds the same best candidate.
__device__ __forceinline__ bool better_candidate(unsigned long long k, uint32_t o, unsigned long long k0, uint32_t o0,
                                                 bool last_level)
{
    if (o == ~0u) return false;
    if (o0 == ~0u) return true;
    return last_level ? o > o0 : (k > k0 || (k == k0 && o < o0));
}

// every lane ends with the warp's best (k, o)
__device__ __forceinline__ void warp_best(unsigned long long& k, uint32_t& o, bool last_level)
{
    for (int d = 16; d; d >>= 1) {
        const unsigned long long k2 = __shfl_xor_sync(kFull, k, d);
        const uint32_t o2 = __shfl_xor_sync(kFull, o, d);
        if (better_candidate(k2, o2, k, o, last_level)) {
            k = k2;
            o = o2;
        }
    }
}

// orientation counts of the eight pieces of a word, in its nibbles
__device__ __forceinline__ uint32_t nibble_counts(uint32_t v)
{
    v -= (v >> 1) & 0x55555555u;
    return (v & 0x33333333u) + ((v >> 2) & 0x33333333u);
}

// Keeps the six smallest (ASC) or largest keys.
template <bool ASC>
__device__ __forceinline__ void keep_six(uint32_t* best, uint32_t v)
{
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        const uint32_t keep = ASC ? min(best[k], v) : max(best[k], v);
        v = ASC ? max(best[k], v) : min(best[k], v);
        best[k] = keep;
    }
}

// Per-pass statistics of the current level (block-wide).  The six smallest and largest
// A[j]-N[j][q] of a piece are found by visiting the infos in order of A: N is at most 4, so
// the visit ends once no later info can enter the list (a scan of all 256 infos for each
// piece and list took most of the statistics' time).
__device__ void level_statistics(GmSmem& sm, uint32_t n, uint32_t nb, uint32_t tid)
{
    const uint32_t lane = tid & 31, warp = tid >> 5;
    for (uint32_t j = warp; j < 256; j += kThreads / 32) {
        uint32_t a = 0;
        if (j < nb) {
            const uint32_t word = sm.X[j][lane];
            const uint32_t x = nibble_counts(word), even = x & 0x0F0F0F0Fu, odd = (x >> 4) & 0x0F0F0F0Fu;
            *reinterpret_cast<uint2*>(&sm.N[j][8 * lane]) =
                make_uint2(__byte_perm(even, odd, 0x5140), __byte_perm(even, odd, 0x7362));
            a = __reduce_add_sync(kFull, __popc(word));
        }
        if (lane == 0) {
            sm.A[j] = static_cast<uint16_t>(a);
            sm.K[j] = j < nb ? (a << 8) | j : ~0u;
        }
    }
    __syncthreads();
    {
        // sums of N: four pieces a word, 16 infos a thread (at most 64 a byte)
        const uint32_t col = tid & 63u, group = tid >> 6;
        uint32_t acc = 0;
        for (uint32_t j = group; j < nb; j += 16) acc += *reinterpret_cast<const uint32_t*>(&sm.N[j][4 * col]);
        sm.part[group][col] = acc;
        // ranks: 64 keys a thread
        const uint32_t j = tid & 255u, from = 64 * (tid >> 8), mine = sm.K[j];
        uint32_t before = 0;
        if (from < nb) {
#pragma unroll 4
            for (uint32_t k = 0; k < 64; k += 4) {
                const uint4 v = *reinterpret_cast<const uint4*>(&sm.K[from + k]);
                before += (v.x < mine) + (v.y < mine) + (v.z < mine) + (v.w < mine);
            }
        }
        sm.rank[tid >> 8][j] = static_cast<uint16_t>(before);
    }
    __syncthreads();
    if (tid < 256) {
        uint32_t s = 0;
        for (uint32_t g = 0; g < 16; ++g) s += (sm.part[g][tid >> 2] >> (8 * (tid & 3u))) & 0xFFu;
        sm.S[tid] = static_cast<uint16_t>(s);
    } else if (tid < 512) {
        const uint32_t j = tid - 256;
        if (j < nb) sm.ord[sm.rank[0][j] + sm.rank[1][j] + sm.rank[2][j] + sm.rank[3][j]] = static_cast<uint8_t>(j);
    } else if (tid < 544) {
        uint32_t a[8], sum = 0;
        bool empty = false;
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) {
            const uint32_t j = 8 * lane + k;
            a[k] = sum;
            sum += sm.A[j];
            empty |= j < nb && sm.A[j] == 0;
        }
        uint32_t x = sum;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(kFull, x, o);
            if (lane >= static_cast<uint32_t>(o)) x += y;
        }
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) sm.cum[8 * lane + k] = x - sum + a[k];
        empty = __any_sync(kFull, empty);
        if (lane == 31) {
            sm.cum[256] = x;
            sm.sumA = x;
            sm.any_empty = empty;
        }
    }
    __syncthreads();
    if (tid < 512) {
        const uint32_t q = tid & 255u;
        uint32_t best[6];
        if (q < n && sm.S[q]) {
            if (tid < 256) {
#pragma unroll
                for (int k = 0; k < 6; ++k) best[k] = ~0u;
                for (uint32_t t = 0; t < nb; ++t) {
                    const uint32_t j = sm.ord[t], a = sm.A[j];
                    if (a >= (best[5] >> 16) + 4) break;
                    keep_six<true>(best, ((a - sm.N[j][q]) << 16) | j);
                }
#pragma unroll
                for (int k = 0; k < 6; ++k) sm.lo[q][k] = best[k];
            } else {
#pragma unroll
                for (int k = 0; k < 6; ++k) best[k] = 0u;
                for (uint32_t t = nb; t-- > 0;) {
                    const uint32_t j = sm.ord[t], a = sm.A[j];
                    if (a + 1 <= (best[5] >> 16)) break;
                    keep_six<false>(best, ((a - sm.N[j][q] + 1) << 16) | j);
                }
#pragma unroll
                for (int k = 0; k < 6; ++k) sm.hi[q][k] = best[k];
            }
        }
    }
    __syncthreads();
}

// What the trials of one position share, in the registers of a group of G lanes.
struct TrialSite {
    uint32_t j[4];      // free neighbours by side (N, E, S, W); 0xFFFF none
    uint32_t x[4];      // this lane's word of their infos, 0 for none
    uint32_t left[4];   // 16-bit pairs: S[q] less this position's and the neighbours' N, of the
                        // lane's pieces (0,2) (4,6) (1,3) (5,7)
    uint32_t sum_a;     // bits of the other positions
};

template <int G>
__device__ __forceinline__ void start_site(const GmSmem& sm, uint32_t nb, uint32_t i, uint32_t width, uint32_t height,
                                           uint32_t lane, TrialSite& t)
{
    const uint32_t pos = sm.position_index[i], px = pos % width, py = pos / width;
    const uint4 s8 = *reinterpret_cast<const uint4*>(&sm.S[8 * lane]);  // (0,1) (2,3) (4,5) (6,7)
    const uint2 ni = *reinterpret_cast<const uint2*>(&sm.N[i][8 * lane]);
    uint2 n = ni;  // bytes: at most 4 a position
    t.sum_a = sm.sumA - sm.A[i];
#pragma unroll
    for (uint32_t s = 0; s < 4; ++s) {
        const bool inside = s == 0 ? py > 0 : s == 1 ? px + 1 < width : s == 2 ? py + 1 < height : px > 0;
        const uint32_t npos = s == 0 ? pos - width : s == 1 ? pos + 1 : s == 2 ? pos + width : pos - 1;
        const uint32_t j = inside ? sm.info_index[npos] : ~0u;
        const bool free = j < nb;
        t.j[s] = free ? j : 0xFFFFu;
        t.x[s] = 0;
        if (free) {
            t.x[s] = sm.X[j][lane];
            const uint2 v = *reinterpret_cast<const uint2*>(&sm.N[j][8 * lane]);
            n.x += v.x;
            n.y += v.y;
            t.sum_a -= sm.A[j];
        }
    }
    // 16-bit pairs, no borrow between halves: S[q] counts every one of these positions
    t.left[0] = __byte_perm(s8.x, s8.y, 0x5410) - __byte_perm(n.x, 0u, 0x4240);
    t.left[1] = __byte_perm(s8.z, s8.w, 0x5410) - __byte_perm(n.y, 0u, 0x4240);
    t.left[2] = __byte_perm(s8.x, s8.y, 0x7632) - __byte_perm(n.x, 0u, 0x4341);
    t.left[3] = __byte_perm(s8.z, s8.w, 0x7632) - __byte_perm(n.y, 0u, 0x4341);
}

struct Trial {
    bool valid;
    uint32_t total, mn, mx;
};

template <int G>
__device__ __forceinline__ uint32_t group_add(uint32_t v, uint32_t gmask)
{
    if (G == 32) return __reduce_add_sync(kFull, v);
    for (int o = G / 2; o; o >>= 1) v += __shfl_xor_sync(gmask, v, o);
    return v;
}

// Trial placement of (info i, word wc, bit b) on the current level by a group of lanes.  Mirrors
// the lambdas of remove_invalid_transitions and get_best_candidate.  `taken`: 0xFFFF in the
// 16-bit place of each piece of the lane that is not available (ordered as TrialSite::left).
template <int G>
__device__ __forceinline__ Trial trial(const GmSmem& sm, const TrialSite& t, const uint32_t* taken, uint32_t i,
                                       uint32_t wc, uint32_t b, uint32_t lane, uint32_t gshift, uint32_t gmask)
{
    Trial r{true, 0, ~0u, 0};
    const uint32_t k = b >> 2, p = 8 * wc + k;
    const bool own = lane == wc;
    const uint32_t pm = own ? ~(0xFu << (4 * k)) : kFull;
    const uint32_t c4 = *reinterpret_cast<const uint32_t*>(sm.pieces[p]);
    const uint32_t col = __funnelshift_r(c4, c4, 8 * (b & 3u));  // byte s: colour of side s
    // apply_color_constraints (CUDA_glutton_max.h:531-612)
    uint32_t even = 0, odd = 0, pc01 = 0, pc23 = 0;
#pragma unroll
    for (uint32_t s = 0; s < 4; ++s) {
        const uint32_t c = (col >> (8 * s)) & 0xFFu;
        uint32_t rw = 0;
        if (c && t.j[s] != 0xFFFFu) rw = t.x[s] & sm.cc[c - 1][s][lane] & pm;
        const uint32_t x = nibble_counts(rw);
        even += x & 0x0F0F0F0Fu;
        odd += (x >> 4) & 0x0F0F0F0Fu;
        const uint32_t pc = __popc(rw);
        if (s < 2) pc01 += pc << (16 * s);
        else pc23 += pc << (16 * (s - 2));
    }
    pc01 = group_add<G>(pc01, gmask);
    pc23 = group_add<G>(pc23, gmask);
    uint32_t kept = 0;
#pragma unroll
    for (uint32_t s = 0; s < 4; ++s) {
        if (t.j[s] == 0xFFFFu || !((col >> (8 * s)) & 0xFFu)) continue;
        const uint32_t pc = ((s < 2 ? pc01 : pc23) >> (16 * (s & 1u))) & 0xFFFFu;
        r.valid &= pc != 0;
        kept += pc;
        r.mn = min(r.mn, pc);
        r.mx = max(r.mx, pc);
    }
    // pieces: every available piece other than p needs a place left
    const uint32_t c0 = t.left[0] + __byte_perm(even, 0u, 0x4140), c1 = t.left[1] + __byte_perm(even, 0u, 0x4342);
    const uint32_t c2 = t.left[2] + __byte_perm(odd, 0u, 0x4140), c3 = t.left[3] + __byte_perm(odd, 0u, 0x4342);
    const uint32_t at = own ? 0xFFFFu << (8 * (k & 2u)) : 0u;  // p's half
    const uint32_t m0 = (k & 5u) == 0u ? at : 0u, m1 = (k & 5u) == 4u ? at : 0u;
    const uint32_t m2 = (k & 5u) == 1u ? at : 0u, m3 = (k & 5u) == 5u ? at : 0u;
    const uint32_t lo = __vminu2(__vminu2(c0 | taken[0] | m0, c1 | taken[1] | m1),
                                 __vminu2(c2 | taken[2] | m2, c3 | taken[3] | m3));
    // (a piece that is not available has no bit anywhere: its count is 0)
    const uint32_t hi = __vmaxu2(__vmaxu2(c0 & ~m0, c1 & ~m1), __vmaxu2(c2 & ~m2, c3 & ~m3));
    uint32_t pmin, pmax;
    if (G == 32) {
        pmin = __reduce_min_sync(kFull, min(lo & 0xFFFFu, lo >> 16));
        pmax = __reduce_max_sync(kFull, max(hi & 0xFFFFu, hi >> 16));
    } else {
        // both at once: the minimum, and the maximum as the minimum of its complement
        uint32_t both = min(lo & 0xFFFFu, lo >> 16) | ((0xFFFFu - max(hi & 0xFFFFu, hi >> 16)) << 16);
        for (int o = G / 2; o; o >>= 1) both = __vminu2(both, __shfl_xor_sync(gmask, both, o));
        pmin = both & 0xFFFFu;
        pmax = 0xFFFFu - (both >> 16);
    }
    r.valid &= pmin != 0;
    if (pmin != 0xFFFFu) r.mn = min(r.mn, pmin);
    r.mx = max(r.mx, pmax);
    // what this position and the neighbours leave of S[p], from the lane that holds p
    const uint32_t mine = (k & 1u) ? ((k & 4u) ? t.left[3] : t.left[2]) : ((k & 4u) ? t.left[1] : t.left[0]);
    const uint32_t sum_n = (__shfl_sync(gmask, mine, wc, G) >> (8 * (k & 2u))) & 0xFFFFu;
    // every other free position keeps its info without piece p (apply_simple_mask); the bits of
    // the pieces are the same bits again
    r.total = 2 * (t.sum_a - sum_n + kept);
    // the smallest and the largest of them: the first of the lists that is not this position or a
    // neighbour (lanes 0..5 look at an entry each)
    const uint32_t el = lane < 6 ? sm.lo[p][lane] : ~0u, eh = lane < 6 ? sm.hi[p][lane] : 0u;
    auto other = [&](uint32_t e) {
        const uint32_t j = e & 0xFFFFu;
        return j != i && j != t.j[0] && j != t.j[1] && j != t.j[2] && j != t.j[3];
    };
    const uint32_t bl = (__ballot_sync(gmask, el != ~0u && other(el)) >> gshift) & 63u;
    const uint32_t bh = (__ballot_sync(gmask, eh != 0u && other(eh)) >> gshift) & 63u;
    const uint32_t vl = __shfl_sync(gmask, el, bl ? __ffs(bl) - 1 : 0, G) >> 16;
    const uint32_t vh = __shfl_sync(gmask, eh, bh ? __ffs(bh) - 1 : 0, G) >> 16;
    if (bl) {
        r.valid &= vl != 0;
        r.mn = min(r.mn, vl);
    }
    if (bh) r.mx = max(r.mx, vh - 1u);
    return r;
}

__device__ void load_level(GmSmem& sm, const GmLaunch& P, uint32_t level, uint32_t tid)
{
    const uint32_t S = P.n, nb = S - level;
    const uint32_t* src = P.infos + static_cast<size_t>(tri_base(S, level)) * 32;
    // from L2: in grid mode other blocks wrote most of it
    for (uint32_t k = 4 * tid; k < nb * 32; k += 4 * kThreads)
        *reinterpret_cast<uint4*>(&sm.X[k >> 5][k & 31]) = __ldcg(reinterpret_cast<const uint4*>(src + k));
}

// rows first, first + stride, ... of the level
__device__ void store_level(const GmSmem& sm, const GmLaunch& P, uint32_t level, uint32_t tid, uint32_t first,
                            uint32_t stride)
{
    const uint32_t S = P.n, nb = S - level;
    uint32_t* dst = P.infos + static_cast<size_t>(tri_base(S, level)) * 32;
    for (uint32_t j = first + stride * (tid >> 5); j < nb; j += stride * (kThreads / 32))
        dst[j * 32 + (tid & 31)] = sm.X[j][tid & 31];
}

// CUDA_glutton_max_stack::pop (thread 0); returns the restored info index.
// `owner` (the block that keeps the global search record) also updates it.
__device__ uint32_t pop_state(GmSmem& sm, GmState* st, uint32_t S, bool owner)
{
    const uint32_t level = sm.level;
    const uint32_t last = S - level;
    const uint32_t info = sm.position_index[last];
    const uint32_t played = sm.played[level - 1];
    const uint32_t pos = played & 0xFFu;
    sm.level = level - 1;
    const uint32_t piece = (played >> 8) & 0xFFu;
    sm.avail[piece >> 5] |= 1u << (piece & 31);
    sm.position_index[last] = pos;
    const uint32_t pos2 = sm.position_index[info];
    uint32_t t = sm.info_index[pos];
    sm.info_index[pos] = sm.info_index[pos2];
    sm.info_index[pos2] = t;
    t = sm.position_index[info];
    sm.position_index[info] = sm.position_index[last];
    sm.position_index[last] = t;
    if (owner) st->pops++;
    return info;
}

// CUDA_glutton_max_stack::push (thread 0).
__device__ void push_state(GmSmem& sm, GmState* st, uint32_t S, uint32_t info, uint32_t pos, uint32_t piece, uint32_t o,
                           bool owner)
{
    const uint32_t level = sm.level;
    sm.played[level] = (o << 16) | (piece << 8) | pos;
    sm.avail[piece >> 5] &= ~(1u << (piece & 31));
    const uint32_t nl = level + 1;
    sm.level = nl;
    if (owner) {
        st->played[level] = sm.played[level];
        if (nl > st->max) {
            for (uint32_t l = 0; l <= st->max && l < S; ++l) st->max_played[l] = sm.played[l];
            st->max = nl;
        }
        st->pushes++;
    }
    ++sm.pushes;
    const uint32_t last = S - nl;
    const uint32_t last_pos = sm.position_index[last];
    sm.position_index[info] = info;
    uint32_t t = sm.info_index[pos];
    sm.info_index[pos] = sm.info_index[last_pos];
    sm.info_index[last_pos] = t;
    t = sm.position_index[info];
    sm.position_index[info] = sm.position_index[last];
    sm.position_index[last] = t;
}

// Grid barrier of the cooperative launch (all blocks are resident).  The wait is
// bounded: past the deadline the block flags an error and the barrier reports it.
__device__ bool grid_sync(GmGrid* g, uint32_t nblocks)
{
    __syncthreads();
    __shared__ uint32_t ok_s;
    if (threadIdx.x == 0) {
        uint32_t ok = 1;
        const uint32_t gen = *(volatile uint32_t*)&g->bar_gen;
        __threadfence();
        if (atomicAdd(&g->bar_count, 1u) == nblocks - 1) {
            g->bar_count = 0;
            __threadfence();
            atomicAdd(&g->bar_gen, 1u);
        } else {
            const uint64_t deadline = global_ns() + kBarrierWaitNs;
            while (*(volatile uint32_t*)&g->bar_gen == gen) {
                if (*(volatile int*)&g->error || global_ns() > deadline) {
                    atomicExch(&g->error, 1);
                    ok = 0;
                    break;
                }
            }
        }
        __threadfence();
        ok_s = ok;
    }
    __syncthreads();
    return ok_s != 0;
}

// The pass's candidates from rank r0 to r1, tried by one group of G lanes; returns the group's
// best valid one and marks the invalid ones.
template <bool GRID, int G>
__device__ __forceinline__ void try_candidates(GmSmem& sm, GmGrid* g, uint32_t buf, uint32_t nb, uint32_t width,
                                               uint32_t height, uint32_t r0, uint32_t r1, bool last_level,
                                               unsigned long long& best_key, uint32_t& best_order)
{
    const uint32_t lane = threadIdx.x & (G - 1), gshift = threadIdx.x & 31u & ~(G - 1u);
    const uint32_t gmask = G == 32 ? kFull : ((1u << (G & 31)) - 1u) << gshift;
    uint32_t taken[4];
    {
        const uint32_t av = sm.avail[lane >> 2] >> (8 * (lane & 3u));  // availability of the lane's pieces
        auto gone = [&](uint32_t a, uint32_t c) {
            return ((av >> a) & 1u ? 0u : 0xFFFFu) | ((av >> c) & 1u ? 0u : 0xFFFF0000u);
        };
        taken[0] = gone(0, 2);
        taken[1] = gone(4, 6);
        taken[2] = gone(1, 3);
        taken[3] = gone(5, 7);
    }
    // the info that holds candidate r0
    uint32_t i = 0;
    for (uint32_t step = 128; step; step >>= 1)
        if (i + step < nb && sm.cum[i + step] <= r0) i += step;
    // its word and bit
    uint32_t word = sm.X[i][lane];
    uint32_t skip = r0 - sm.cum[i], w = 0;
    {
        const uint32_t pc = __popc(word);
        uint32_t x = pc;
        for (int o = 1; o < G; o <<= 1) {
            const uint32_t y = __shfl_up_sync(gmask, x, o, G);
            if (lane >= static_cast<uint32_t>(o)) x += y;
        }
        const uint32_t holds = (__ballot_sync(gmask, x > skip) >> gshift);
        w = __ffs(holds) - 1;
        skip -= __shfl_sync(gmask, x - pc, w, G);
    }
    uint32_t todo = (__ballot_sync(gmask, word != 0) >> gshift) & (G == 32 ? kFull : (1u << (G & 31)) - 1u);
    todo &= ~0u << w;
    uint32_t bits = __shfl_sync(gmask, word, w, G);
    for (; skip; --skip) bits &= bits - 1;
    TrialSite site;
    start_site<G>(sm, nb, i, width, height, lane, site);
    for (uint32_t r = r0; r < r1; ++r) {
        if (!bits) {
            todo &= todo - 1;
            if (!todo) {
                ++i;
                word = sm.X[i][lane];
                todo = (__ballot_sync(gmask, word != 0) >> gshift) & (G == 32 ? kFull : (1u << (G & 31)) - 1u);
                start_site<G>(sm, nb, i, width, height, lane, site);
            }
            w = __ffs(todo) - 1;
            bits = __shfl_sync(gmask, word, w, G);
        }
        const uint32_t b = __ffs(bits) - 1;
        bits &= bits - 1;
        const Trial t = trial<G>(sm, site, taken, i, w, b, lane, gshift, gmask);
        const uint32_t order = (i << 10) | (w << 5) | b;
        if (!t.valid) {
            if (lane == 0) {
                if (GRID) {
                    atomicOr(&g->inval[buf][i][w], 1u << b);
                    g->any_invalid[buf] = 1;
                } else {
                    atomicOr(&sm.inval[i][w], 1u << b);
                    sm.any_invalid = 1;
                }
            }
        } else {
            const unsigned long long key = (static_cast<unsigned long long>(t.total) << 32) | ((t.mx << 16) + t.mn);
            if (better_candidate(key, order, best_key, best_order, last_level)) {
                best_key = key;
                best_order = order;
            }
        }
    }
}

// One glutton max search.  GRID = false: one block does everything.  GRID = true:
// every block of a cooperative launch keeps a copy of the level and makes the same
// decisions; the candidate trials of each validity pass are shared out over the groups
// of all blocks, results meet in global memory (triple-buffered per pass, one grid barrier per
// pass), and block 0 keeps the global search record.
template <bool GRID, int G>
__global__ void __launch_bounds__(kThreads, 1) gm_kernel(GmLaunch P)
{
    extern __shared__ __align__(16) unsigned char gm_raw[];
    GmSmem& sm = *reinterpret_cast<GmSmem*>(gm_raw);
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t S = P.n, height = P.n / P.width;
    GmState* st = P.state;
    GmGrid* g = P.grid;
    const bool owner = !GRID || blockIdx.x == 0;
    const uint32_t nblocks = GRID ? gridDim.x : 1u, block = GRID ? blockIdx.x : 0u;
    uint32_t pass_no = 0;  // grid mode: passes so far (selects the exchange buffer)
    bool grid_failed = false;
    // grid mode: rows of a level were stored since the last barrier (every block's share)
    bool stored = false;
    auto load_popped = [&](uint32_t at) {
        if (GRID && stored) {
            if (!grid_sync(g, nblocks)) grid_failed = true;
            stored = false;
        }
        if (!grid_failed) load_level(sm, P, at, tid);
    };
    for (uint32_t k = tid; k < 256 * 4; k += kThreads) sm.pieces[k >> 2][k & 3] = P.pieces[k];
    for (uint32_t k = tid; k < P.ncolours * 4 * 32; k += kThreads) (&sm.cc[0][0][0])[k] = P.cc[k];
    for (uint32_t k = tid; k < 256; k += kThreads) {
        sm.position_index[k] = st->position_index[k];
        sm.info_index[k] = st->info_index[k];
        sm.played[k] = st->played[k];
    }
    if (tid < 8) sm.avail[tid] = st->avail[tid];
    if (tid == 0) {
        sm.level = st->level;
        sm.new_level = st->new_level;
        sm.pop_index = st->pop_index;
        sm.stop = 0;
        sm.trials = st->trials;
        sm.pushes = st->pushes;
    }
    __syncthreads();
    load_level(sm, P, sm.level, tid);
    __syncthreads();
    const uint64_t deadline = P.timeout_ns ? global_ns() + P.timeout_ns : 0;

    for (;;) {
        const uint32_t level = sm.level;
        if (level >= S) break;  // full board (level == S) or exhausted (wrapped below 0)
        // the budgets are counted alike by every block; the clock is block 0's, left in sm.stop by
        // the passes of the level before
        if (tid == 0) {
            if ((P.push_budget && sm.pushes >= P.push_budget) ||
                (P.placement_budget && sm.trials + sm.pushes >= P.placement_budget))
                sm.stop = 1;
            if (!GRID && deadline && global_ns() > deadline) sm.stop = 1;
        }
        __syncthreads();
        if (sm.stop) break;
        const uint32_t nb = S - level;
        // a popped level whose tried candidate was its last one pops again
        if (!sm.new_level) {
            const uint32_t any = __syncthreads_or(tid < 32 && sm.X[sm.pop_index][tid] != 0);
            if (!any) {
                __syncthreads();
                if (tid == 0) {
                    if (level == 0) sm.level = ~0u;
                    else sm.pop_index = pop_state(sm, st, S, owner);
                    sm.new_level = 0;
                }
                __syncthreads();
                if (sm.level < S) load_popped(sm.level);
                if (grid_failed) break;
                __syncthreads();
                continue;
            }
        }
        if (owner && tid == 0) st->levels++;
        // ---- validity fixpoint and scores ----
        bool failed = false;
        for (;;) {
            level_statistics(sm, S, nb, tid);
            if (sm.any_empty) {
                failed = true;
                break;
            }
            const uint32_t buf = pass_no % 3;
            if (!GRID) {
                for (uint32_t k = tid; k < nb * 32; k += kThreads) sm.inval[k >> 5][k & 31] = 0;
            }
            if (tid == 0) {
                sm.any_invalid = 0;
                sm.trials += sm.sumA;  // every candidate is tried
                if (owner) {
                    st->passes++;
                    if (GRID) g->stop[buf] = deadline && global_ns() > deadline;
                }
            }
            __syncthreads();
            unsigned long long best_key = 0;
            uint32_t best_order = ~0u;
            const bool last_level = level == S - 1;
            {
                const uint32_t groups = nblocks * (kThreads / G);
                // neighbouring ranges go to different blocks
                const uint32_t me = (tid / G) * nblocks + block;
                const uint32_t r0 = static_cast<uint32_t>(static_cast<uint64_t>(sm.sumA) * me / groups);
                const uint32_t r1 = static_cast<uint32_t>(static_cast<uint64_t>(sm.sumA) * (me + 1) / groups);
                if (r0 < r1)
                    try_candidates<GRID, G>(sm, g, buf, nb, P.width, height, r0, r1, last_level, best_key, best_order);
            }
            __syncwarp();
            if (G < 32) warp_best(best_key, best_order, last_level);
            if (lane == 0) {
                sm.warp_key[warp] = best_key;
                sm.warp_order[warp] = best_order;
            }
            __syncthreads();
            // this block's best, reduced by warp 0 (a strict total order: any reduction
            // order gives the same result)
            if (warp == 0) {
                unsigned long long k0 = sm.warp_key[lane];
                uint32_t o0 = sm.warp_order[lane];
                warp_best(k0, o0, last_level);
                if (lane == 0) {
                    if (GRID) {
                        g->blk_key[buf][blockIdx.x] = k0;
                        g->blk_order[buf][blockIdx.x] = o0;
                    } else {
                        sm.best_order = o0;
                    }
                }
            }
            if (GRID) {
                if (!grid_sync(g, nblocks)) {
                    grid_failed = true;
                    break;
                }
                stored = false;
                // the buffer of the pass before last is free again: every block clears its rows
                const uint32_t old = (pass_no + 2) % 3;
                for (uint32_t j = block + nblocks * warp; j < S; j += nblocks * (kThreads / 32))
                    g->inval[old][j][lane] = 0;
                if (block == 0 && tid == 0) g->any_invalid[old] = 0;
                if (warp == 0) {
                    // the blocks' bests, 32 at a time (the loads overlap instead of
                    // waiting on L2 one block after another)
                    unsigned long long k0 = 0;
                    uint32_t o0 = ~0u;
                    for (uint32_t b2 = lane; b2 < nblocks; b2 += 32) {
                        const uint32_t o = *(volatile uint32_t*)&g->blk_order[buf][b2];
                        const unsigned long long k = *(volatile unsigned long long*)&g->blk_key[buf][b2];
                        if (better_candidate(k, o, k0, o0, last_level)) {
                            k0 = k;
                            o0 = o;
                        }
                    }
                    warp_best(k0, o0, last_level);
                    if (lane == 0) {
                        sm.any_invalid = *(volatile uint32_t*)&g->any_invalid[buf];
                        sm.best_order = o0;
                        sm.stop = *(volatile uint32_t*)&g->stop[buf];
                    }
                }
                ++pass_no;
            }
            __syncthreads();
            if (!sm.any_invalid) break;
            if (GRID) {
                for (uint32_t k = 4 * tid; k < nb * 32; k += 4 * kThreads) {
                    const uint4 v = __ldcg(reinterpret_cast<const uint4*>(&g->inval[buf][k >> 5][k & 31]));
                    uint4& x = *reinterpret_cast<uint4*>(&sm.X[k >> 5][k & 31]);
                    x = make_uint4(x.x & ~v.x, x.y & ~v.y, x.z & ~v.z, x.w & ~v.w);
                }
            } else {
                for (uint32_t k = tid; k < nb * 32; k += kThreads) sm.X[k >> 5][k & 31] &= ~sm.inval[k >> 5][k & 31];
            }
            __syncthreads();
        }
        if (grid_failed) break;
        if (failed || sm.best_order == ~0u) {
            // remove_invalid_transitions failed or no candidate: pop
            __syncthreads();
            if (tid == 0) {
                if (level == 0) sm.level = ~0u;
                else sm.pop_index = pop_state(sm, st, S, owner);
                sm.new_level = 0;
            }
            __syncthreads();
            if (sm.level < S) load_popped(sm.level);
            if (grid_failed) break;
            __syncthreads();
            continue;
        }
        // ---- apply_best_candidate ----
        const uint32_t bi = sm.best_order >> 10, bw = (sm.best_order >> 5) & 31u, bb = sm.best_order & 31u;
        const uint32_t piece = 8 * bw + bb / 4, o = bb & 3u;
        const uint32_t pos = sm.position_index[bi];
        if (tid == 0) sm.X[bi][bw] &= ~(1u << bb);
        __syncthreads();
        // the level keeps its remaining candidates for a later pop.  In grid mode each block
        // writes its share, and a pop reads the level after a barrier.
        store_level(sm, P, level, tid, block, nblocks);
        stored = true;
        const uint32_t pm_word = ~(0xFu << (4 * (bb / 4)));
        // the next level moves the last info into the chosen slot; an empty
        // result there stops the reference's apply before its push
        const bool copy_last = bi < nb - 1 && level < S - 1;
        const uint32_t last_any =
            copy_last ? __syncthreads_or(tid < 32 && (sm.X[nb - 1][tid] & (tid == bw ? pm_word : kFull)) != 0) : 1u;
        if (!last_any) {
            if (tid == 0) sm.new_level = 1;
            __syncthreads();
            continue;
        }
        __syncthreads();
        // next level in place: X[j] &= pm for j < nb-1, X[bi] = X[nb-1] & pm
        for (uint32_t k = tid; k < (nb - 1) * 32; k += kThreads) {
            const uint32_t j = k >> 5, w = k & 31;
            const uint32_t m = w == bw ? pm_word : kFull;
            if (j == bi) sm.X[j][w] = sm.X[nb - 1][w] & m;
            else sm.X[j][w] &= m;
        }
        __syncthreads();
        if (tid == 0) push_state(sm, st, S, bi, pos, piece, o, owner);
        __syncthreads();
        // colour constraints of the placed piece on its free neighbours
        if (warp == 0) {
            const uint32_t nl = sm.level, nbn = S - nl;
            const int off[4] = {-static_cast<int>(P.width), 1, static_cast<int>(P.width), -1};
            bool invalid = false;
            for (uint32_t s2 = 0; s2 < 4 && !invalid; ++s2) {
                const uint32_t col = sm.pieces[piece][(s2 + o) & 3u];
                if (!col) continue;
                const uint32_t npos = static_cast<uint32_t>(static_cast<int>(pos) + off[s2]);
                const uint32_t j = sm.info_index[npos];
                if (j >= nbn) continue;
                const uint32_t r = sm.X[j][lane] & sm.cc[col - 1][s2][lane];
                if (!__any_sync(kFull, r)) {
                    invalid = true;
                    break;
                }
                sm.X[j][lane] = r;
            }
            if (lane == 0) sm.apply_failed = invalid;
        }
        __syncthreads();
        if (sm.apply_failed) {
            __syncthreads();
            if (tid == 0) pop_state(sm, st, S, owner);
            __syncthreads();
            load_popped(sm.level);
            if (grid_failed) break;
        }
        if (tid == 0) sm.new_level = 1;
        __syncthreads();
    }
    // write the search state back (the owner block)
    __syncthreads();
    if (!owner) return;
    if (tid == 0) {
        const uint32_t level = sm.level;
        st->level = level;
        st->new_level = sm.new_level;
        st->pop_index = sm.pop_index;
        st->trials = sm.trials;
        st->status = grid_failed ? 3 : (level == S ? 0 : (level > S ? 2 : 1));
    }
    if (sm.level < S) store_level(sm, P, sm.level, tid, 0, 1);
    for (uint32_t k = tid; k < 256; k += kThreads) {
        st->position_index[k] = sm.position_index[k];
        st->info_index[k] = sm.info_index[k];
    }
    if (tid < 8) st->avail[tid] = sm.avail[tid];
}

}  // namespace

size_t gm_smem_bytes() { return sizeof(GmSmem); }

namespace {

// lanes of a trial's group: the words that hold pieces
template <bool GRID>
const void* gm_symbol(uint32_t n)
{
    if (n <= 64) return reinterpret_cast<const void*>(&gm_kernel<GRID, 8>);
    if (n <= 128) return reinterpret_cast<const void*>(&gm_kernel<GRID, 16>);
    return reinterpret_cast<const void*>(&gm_kernel<GRID, 32>);
}

}  // namespace

cudaError_t launch_gm(const GmLaunch& P, cudaStream_t stream)
{
    const size_t smem = sizeof(GmSmem);
    const void* fn = gm_symbol<false>(P.n);
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return e;
    GmLaunch copy = P;
    void* args[] = {&copy};
    return cudaLaunchKernel(fn, dim3(1), dim3(kThreads), args, smem, stream);
}

cudaError_t launch_gm_grid(const GmLaunch& P, uint32_t blocks, cudaStream_t stream)
{
    const size_t smem = sizeof(GmSmem);
    const void* fn = gm_symbol<true>(P.n);
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kThreads, smem);
    if (e != cudaSuccess) return e;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (per_sm < 1 || blocks > static_cast<uint32_t>(per_sm * sms) || blocks > kMaxGridBlocks || !blocks)
        return cudaErrorCooperativeLaunchTooLarge;
    GmLaunch copy = P;
    void* args[] = {&copy};
    return cudaLaunchCooperativeKernel(fn, dim3(blocks), dim3(kThreads), args, smem, stream);
}

}  // namespace emp
