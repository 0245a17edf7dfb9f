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
// A trial is made by T threads (a power of two: as many as the pass leaves a candidate), each over
// every T-th word of eight pieces, which shuffles then combine.  A thread treats a word's
// pieces as bit and byte fields: the orientations the neighbours keep are counted in nibbles,
// added as bytes to what position and neighbours take from S (M, worked out once a pass for
// each position), and compared as 16-bit pairs.  The candidates of a pass are dealt out evenly by
// rank; each thread finds its own.
//
// What bounds it: instructions, of the trials (about 85 a word of eight pieces) and of the statistics
// that every block repeats in each pass (16x16, 20 pushes: ALU pipe 65 %, issue slots 58 % busy, 30.7
// lanes in an instruction), and the block barriers between the steps of a pass (the top stall).  Measured on a B200, whole calls: 16x16
// (5/17 colours, 300 pushes, 148 blocks) 165 ms with a warp a trial, shuffles for every sum,
// full scans for the lists and a work counter; 42 ms with a group of lanes a trial, 320
// instructions in each lane; 28 ms now, 22 us a pass of 45 000 trials.  8x8 on one block (150
// pushes): 162, 21 and 12 ms.
#include "emp_gm.h"

#include <cuda_runtime.h>

namespace emp {

namespace {

constexpr int kThreads = 1024;
constexpr unsigned kFull = 0xFFFFFFFFu;
constexpr uint64_t kBarrierWaitNs = 5000000000ull;  // 5 s: far beyond one validity pass

constexpr uint32_t kXs = 33;       // words of a row of infos, padded: rows fall on different banks

struct GmSmem {
    alignas(16) uint32_t X[256][kXs];  // infos of the current level
    alignas(16) uint2 N[256][kXs];     // orientations left of the pieces of a word, a byte each: pieces
                                       // 0,2,4,6 in x, 1,3,5,7 in y.  During the trials of the one-block
                                       // search: the candidates found invalid
    alignas(16) uint2 M[256][kXs];     // 32 less N of info i and of its free neighbours, as N
    uint32_t cc[4][32][kXs];           // colour constraints by side and colour
    alignas(16) uint16_t Sp[32][8];    // S of the pieces (0,2) (4,6) (1,3) (5,7) of a word; 0x8000 for
                                       // pieces that are not available
    uint32_t lo[256][6];       // per piece q: six smallest (A[j]-N[j][q]) << 16 | j, ~0 empty
    uint32_t hi[256][6];       // per piece q: six largest (A[j]-N[j][q]+1) << 16 | j, 0 empty
    alignas(16) uint32_t K[256];  // A[j] << 8 | j, ~0 past the last info
    uint32_t part[16][64];     // partial sums of N
    uint32_t cum[1024];        // candidates before each quarter of each info's words
    ushort4 nbr[256];          // free neighbours' infos by side (N, E, S, W); 0xFFFF none
    uint32_t near_bits[256];   // bits of info i and its free neighbours
    uint16_t A[256];           // bits of info j
    uint16_t S[256];           // sum over j of N[j][q]
    uint16_t rank[4][256];     // partial ranks of K[j]
    alignas(16) uint32_t sorted[256];  // K in ascending order, ~0 past the last info
    alignas(4) uint8_t pieces[256][4];
    uint32_t position_index[256];
    uint32_t info_index[256];
    uint32_t played[256];      // this block's copy of the played stack
    uint32_t max_played[256];  // ... when most pieces were placed
    uint32_t avail[8];
    unsigned long long warp_key[32];
    uint32_t warp_order[32];
    uint32_t warp_bits[32];    // candidates of the infos of each warp, then of the warps before
    unsigned long long trials, pushes, pops, passes, levels;  // of the search, counted alike by every block
    uint32_t max, new_max;     // most pieces placed; 1: by the last push
    uint32_t sumA;
    uint32_t any_invalid;
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

__device__ __forceinline__ uint32_t min2(uint32_t a, uint32_t b)  // of 16-bit pairs
{
    uint32_t r;
    asm("min.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t max2(uint32_t a, uint32_t b)  // of signed ones
{
    uint32_t r;
    asm("max.s16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
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

// Candidate of rank r: info << 10 | word << 5 | bit.
__device__ __forceinline__ uint32_t candidate_of_rank(const GmSmem& sm, uint32_t r)
{
    uint32_t q = 0;  // the quarter of an info's words that holds it
#pragma unroll
    for (uint32_t step = 512; step; step >>= 1) q += sm.cum[q + step] <= r ? step : 0u;
    r -= sm.cum[q];
    const uint32_t j = q >> 2;
    uint32_t w = 8 * (q & 3u), word = sm.X[j][w];
    for (uint32_t c; (c = __popc(word)) <= r; r -= c) word = sm.X[j][++w];
    uint32_t b = 0;  // the r-th set bit of the word
#pragma unroll
    for (uint32_t half = 16; half; half >>= 1) {
        const uint32_t c = __popc((word >> b) & ((1u << half) - 1u));
        if (c <= r) {
            r -= c;
            b += half;
        }
    }
    return (j << 10) | (w << 5) | b;
}

// Per-pass statistics of the current level (block-wide).  Returns whether an info is empty.  The six
// smallest and largest A[j]-N[j][q] of a piece are found by visiting the infos in order of A: N is at
// most 4, so the visit ends once no later info can enter the list (a scan of all 256 infos for each
// piece and list took most of the statistics' time).
__device__ bool level_statistics(GmSmem& sm, uint32_t n, uint32_t nb, uint32_t width, uint32_t tid)
{
    const uint32_t lane = tid & 31, warp = tid >> 5, j = tid >> 2, w0 = 8 * (tid & 3u);
    uint32_t bits = 0;
    if (j < nb) {
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) {
            const uint32_t word = sm.X[j][w0 + k], x = nibble_counts(word);
            sm.N[j][w0 + k] = make_uint2(x & 0x0F0F0F0Fu, (x >> 4) & 0x0F0F0F0Fu);
            bits += __popc(word);
        }
    }
    uint32_t a = bits + __shfl_xor_sync(kFull, bits, 1);
    a += __shfl_xor_sync(kFull, a, 2);
    uint32_t upto = bits;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, upto, o);
        if (lane >= static_cast<uint32_t>(o)) upto += y;
    }
    if (lane == 31) sm.warp_bits[warp] = upto;
    if (!(tid & 3u)) {
        sm.A[j] = static_cast<uint16_t>(a);
        sm.K[j] = j < nb ? (a << 8) | j : ~0u;
    }
    if (__syncthreads_or(j < nb && a == 0)) return true;
    if (warp == 0) {
        const uint32_t v = sm.warp_bits[lane];
        uint32_t x = v;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(kFull, x, o);
            if (lane >= static_cast<uint32_t>(o)) x += y;
        }
        sm.warp_bits[lane] = x - v;
        if (lane == 31) sm.sumA = x;
    }
    {
        // sums of N: four pieces a word, 16 infos a thread (at most 64 a byte)
        const uint32_t col = tid & 63u, group = tid >> 6;
        uint32_t acc = 0;
        for (uint32_t i = group; i < nb; i += 16) acc += reinterpret_cast<const uint32_t*>(sm.N[i])[col];
        sm.part[group][col] = acc;
        // ranks: 64 keys a thread
        const uint32_t i = tid & 255u, from = 64 * (tid >> 8), key = sm.K[i];
        uint32_t less = 0;
        if (from < nb) {
#pragma unroll 4
            for (uint32_t k = 0; k < 64; k += 4) {
                const uint4 v = *reinterpret_cast<const uint4*>(&sm.K[from + k]);
                less += (v.x < key) + (v.y < key) + (v.z < key) + (v.w < key);
            }
        }
        sm.rank[tid >> 8][i] = static_cast<uint16_t>(less);
    }
    if (j < nb) {
        // this info's free neighbours, and what it and they take from S
        const uint32_t pos = sm.position_index[j], px = pos % width;
        uint32_t at[4], near = a;
#pragma unroll
        for (uint32_t s = 0; s < 4; ++s) {
            const bool inside = s == 0 ? pos >= width : s == 1 ? px + 1 < width : s == 2 ? pos + width < n : px > 0;
            const uint32_t npos = s == 0 ? pos - width : s == 1 ? pos + 1 : s == 2 ? pos + width : pos - 1;
            const uint32_t q = inside ? sm.info_index[npos] : ~0u;
            at[s] = q < nb ? q : 0xFFFFu;
            near += q < nb ? sm.A[q] : 0u;
        }
        if (!(tid & 3u)) {
            sm.nbr[j] = make_ushort4(static_cast<uint16_t>(at[0]), static_cast<uint16_t>(at[1]),
                                     static_cast<uint16_t>(at[2]), static_cast<uint16_t>(at[3]));
            sm.near_bits[j] = near;
        }
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) {
            uint2 m = sm.N[j][w0 + k];
#pragma unroll
            for (uint32_t s = 0; s < 4; ++s) {
                if (at[s] != 0xFFFFu) {
                    const uint2 v = sm.N[at[s]][w0 + k];
                    m.x += v.x;
                    m.y += v.y;
                }
            }
            sm.M[j][w0 + k] = make_uint2(0x20202020u - m.x, 0x20202020u - m.y);
        }
    }
    __syncthreads();
    if (tid < 256) {
        const uint32_t k = tid & 7u;
        uint32_t s = 0;
        for (uint32_t g = 0; g < 16; ++g) s += (sm.part[g][2 * (tid >> 3) + (k & 1u)] >> (8 * (k >> 1))) & 0xFFu;
        sm.S[tid] = static_cast<uint16_t>(s);
        const bool available = (sm.avail[tid >> 5] >> (tid & 31)) & 1u;
        sm.Sp[tid >> 3][4 * (k & 1u) + 2 * (k >> 2) + ((k >> 1) & 1u)] = static_cast<uint16_t>(available ? s : 0x8000u);
    } else if (tid < 512) {
        const uint32_t i = tid - 256;
        if (i < nb) sm.sorted[sm.rank[0][i] + sm.rank[1][i] + sm.rank[2][i] + sm.rank[3][i]] = sm.K[i];
        else sm.sorted[i] = ~0u;
    }
    sm.cum[tid] = sm.warp_bits[warp] + upto - bits;
    __syncthreads();
    if (tid < 512) {
        const uint32_t q = tid & 255u;
        const uint32_t byte = 8 * (q >> 3) + 4 * (q & 1u) + ((q & 7u) >> 1);  // of a row of N
        uint32_t best[6];
        if (q < n && sm.S[q]) {
            // four infos at a time, so that their loads overlap
            if (tid < 256) {
#pragma unroll
                for (int k = 0; k < 6; ++k) best[k] = ~0u;
                for (uint32_t t = 0; t < nb; t += 4) {
                    const uint4 v = *reinterpret_cast<const uint4*>(&sm.sorted[t]);
                    if ((v.x >> 8) >= (best[5] >> 16) + 4) break;
                    const uint32_t key[4] = {v.x, v.y, v.z, v.w};
                    uint32_t c[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) c[k] = reinterpret_cast<const uint8_t*>(sm.N[key[k] & 0xFFu])[byte];
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        keep_six<true>(best, key[k] == ~0u ? ~0u : (((key[k] >> 8) - c[k]) << 16) | (key[k] & 0xFFu));
                }
#pragma unroll
                for (int k = 0; k < 6; ++k) sm.lo[q][k] = best[k];
            } else {
#pragma unroll
                for (int k = 0; k < 6; ++k) best[k] = 0u;
                for (uint32_t t = (nb + 3) & ~3u; t;) {
                    t -= 4;
                    const uint4 v = *reinterpret_cast<const uint4*>(&sm.sorted[t]);
                    const uint32_t top = v.w != ~0u ? v.w : v.z != ~0u ? v.z : v.y != ~0u ? v.y : v.x;
                    if ((top >> 8) + 1 <= (best[5] >> 16)) break;
                    const uint32_t key[4] = {v.x, v.y, v.z, v.w};
                    uint32_t c[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) c[k] = reinterpret_cast<const uint8_t*>(sm.N[key[k] & 0xFFu])[byte];
#pragma unroll
                    for (int k = 3; k >= 0; --k)
                        keep_six<false>(best, key[k] == ~0u ? 0u : (((key[k] >> 8) - c[k] + 1) << 16) | (key[k] & 0xFFu));
                }
#pragma unroll
                for (int k = 0; k < 6; ++k) sm.hi[q][k] = best[k];
            }
        }
    }
    __syncthreads();
    return false;
}

// Trial placement of candidate `code` on the current level by T threads, the sub-th of which this
// is.  Mirrors the lambdas of remove_invalid_transitions and get_best_candidate: the placement is
// valid when the smallest count, over free positions and available pieces, is not 0
// (*smallest).  Returns get_best_candidate's score.
__device__ __forceinline__ unsigned long long trial(const GmSmem& sm, uint32_t code, uint32_t words, uint32_t T,
                                                    uint32_t sub, uint32_t* smallest)
{
    const uint32_t i = code >> 10, wp = (code >> 5) & 31u, b = code & 31u, k = b >> 2, p = 8 * wp + k;
    const ushort4 nb4 = sm.nbr[i];
    const uint32_t at[4] = {nb4.x, nb4.y, nb4.z, nb4.w};
    const uint32_t c4 = *reinterpret_cast<const uint32_t*>(sm.pieces[p]);
    const uint32_t col = __funnelshift_r(c4, c4, 8 * (b & 3u));  // byte s: colour of side s
    // apply_color_constraints (CUDA_glutton_max.h:531-612): rows of the neighbours' infos and
    // of the constraints.  A side without a free neighbour reads row 0 and keeps nothing.
    const uint32_t* x[4];
    const uint32_t* m[4];
    uint32_t on[4];
#pragma unroll
    for (uint32_t s = 0; s < 4; ++s) {
        const uint32_t c = (col >> (8 * s)) & 0xFFu;
        const bool free = at[s] != 0xFFFFu && c;
        on[s] = free ? kFull : 0u;
        x[s] = sm.X[free ? at[s] : 0u];
        m[s] = sm.cc[s][free ? c - 1 : 0u];
    }
    // the piece itself is taken from every info and is not among the pieces that need a place
    const uint32_t half = 0x8000u << (8 * (k & 2u));
    const uint32_t h0 = (k & 5u) == 0u ? half : 0u, h1 = (k & 5u) == 4u ? half : 0u;
    const uint32_t h2 = (k & 5u) == 1u ? half : 0u, h3 = (k & 5u) == 5u ? half : 0u;
    uint32_t lo = 0xFFFFFFFFu, hi = 0x80008000u, pc01 = 0, pc23 = 0;
#pragma unroll 2
    for (uint32_t w = sub; w < words; w += T) {
        const uint32_t own = w == wp ? kFull : 0u, pm = ~((0xFu << (4 * k)) & own);
        const uint32_t r0 = x[0][w] & m[0][w] & (on[0] & pm), r1 = x[1][w] & m[1][w] & (on[1] & pm);
        const uint32_t r2 = x[2][w] & m[2][w] & (on[2] & pm), r3 = x[3][w] & m[3][w] & (on[3] & pm);
        pc01 += __popc(r0) + (__popc(r1) << 16);
        pc23 += __popc(r2) + (__popc(r3) << 16);
        // two neighbours keep at most 8 orientations of a piece: their counts share a nibble
        const uint32_t y01 = nibble_counts(r0) + nibble_counts(r1), y23 = nibble_counts(r2) + nibble_counts(r3);
        const uint2 mm = sm.M[i][w];
        const uint32_t even = mm.x + (y01 & 0x0F0F0F0Fu) + (y23 & 0x0F0F0F0Fu);
        const uint32_t odd = mm.y + ((y01 >> 4) & 0x0F0F0F0Fu) + ((y23 >> 4) & 0x0F0F0F0Fu);
        // every available piece other than p needs a place left: 32 + its count in 16 bits, at
        // least 0x8000 for the others
        const uint4 sp = *reinterpret_cast<const uint4*>(sm.Sp[w]);
        const uint32_t c0 = (sp.x | (h0 & own)) + __byte_perm(even, 0u, 0x4140);
        const uint32_t c1 = (sp.y | (h1 & own)) + __byte_perm(even, 0u, 0x4342);
        const uint32_t c2 = (sp.z | (h2 & own)) + __byte_perm(odd, 0u, 0x4140);
        const uint32_t c3 = (sp.w | (h3 & own)) + __byte_perm(odd, 0u, 0x4342);
        lo = min2(lo, min2(min2(c0, c1), min2(c2, c3)));
        hi = max2(hi, max2(max2(c0, c1), max2(c2, c3)));
    }
    for (uint32_t d = T >> 1; d; d >>= 1) {
        pc01 += __shfl_xor_sync(kFull, pc01, d);
        pc23 += __shfl_xor_sync(kFull, pc23, d);
        lo = min2(lo, __shfl_xor_sync(kFull, lo, d));
        hi = max2(hi, __shfl_xor_sync(kFull, hi, d));
    }
    const uint32_t plo = min(lo & 0xFFFFu, lo >> 16);
    const int phi = max(static_cast<int16_t>(hi & 0xFFFFu), static_cast<int16_t>(hi >> 16));
    uint32_t mn = plo < 0x8000u ? plo - 32 : ~0u, mx = phi >= 32 ? static_cast<uint32_t>(phi) - 32 : 0u, kept = 0;
#pragma unroll
    for (uint32_t s = 0; s < 4; ++s) {
        const uint32_t pc = ((s < 2 ? pc01 : pc23) >> (16 * (s & 1u))) & 0xFFFFu;  // 0 on a side without neighbour
        kept += pc;
        mx = max(mx, pc);
        mn = min(mn, pc | ~on[s]);
    }
    // every other free position keeps its info without piece p (apply_simple_mask): the smallest
    // and the largest are the first of the lists that are not this position or a neighbour
    auto other = [&](uint32_t e) {
        const uint32_t q = e & 0xFFFFu;
        return q != i && q != at[0] && q != at[1] && q != at[2] && q != at[3];
    };
#pragma unroll 1
    for (uint32_t r = 0; r < 6; ++r) {
        const uint32_t e = sm.lo[p][r];
        if (e == ~0u) break;
        if (other(e)) {
            mn = min(mn, e >> 16);
            break;
        }
    }
#pragma unroll 1
    for (uint32_t r = 0; r < 6; ++r) {
        const uint32_t e = sm.hi[p][r];
        if (e == 0u) break;
        if (other(e)) {
            mx = max(mx, (e >> 16) - 1u);
            break;
        }
    }
    *smallest = mn;
    // what this position and the neighbours leave of S[p]
    const uint2 mp = sm.M[i][wp];
    const uint32_t sum_n = sm.S[p] - (32 - ((((k & 1u) ? mp.y : mp.x) >> (8 * (k >> 1))) & 0xFFu));
    // the bits of the pieces are the bits of the positions again
    const uint32_t total = 2 * (sm.sumA - sm.near_bits[i] - sum_n + kept);
    return (static_cast<unsigned long long>(total) << 32) | ((mx << 16) + mn);
}

__device__ void load_level(GmSmem& sm, const GmLaunch& P, uint32_t level, uint32_t tid)
{
    const uint32_t S = P.n, nb = S - level;
    const uint32_t* src = P.infos + static_cast<size_t>(tri_base(S, level)) * 32;
    // from L2: in grid mode other blocks wrote most of it
    for (uint32_t k = 4 * tid; k < nb * 32; k += 4 * kThreads) {
        const uint4 v = __ldcg(reinterpret_cast<const uint4*>(src + k));
        uint32_t* x = &sm.X[k >> 5][k & 31];
        x[0] = v.x;
        x[1] = v.y;
        x[2] = v.z;
        x[3] = v.w;
    }
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
__device__ uint32_t pop_state(GmSmem& sm, uint32_t S)
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
    ++sm.pops;
    return info;
}

// CUDA_glutton_max_stack::push (thread 0).
__device__ void push_state(GmSmem& sm, uint32_t S, uint32_t info, uint32_t pos, uint32_t piece, uint32_t o)
{
    const uint32_t level = sm.level;
    sm.played[level] = (o << 16) | (piece << 8) | pos;
    sm.avail[piece >> 5] &= ~(1u << (piece & 31));
    const uint32_t nl = level + 1;
    sm.level = nl;
    sm.new_max = nl > sm.max;
    if (nl > sm.max) sm.max = nl;
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

// Grid barrier of the cooperative launch (all blocks are resident): every block adds its arrival
// and its flags to one counter, and the value that completes the count tells every block
// whether any block had the flag.  Counters are used in turn and cleared a barrier later (the
// caller's part).  The wait is bounded: past the deadline the block flags an error and the barrier
// reports it.
constexpr uint32_t kArriveInvalid = 1u << 16, kArriveStop = 1u << 31;

__device__ bool grid_sync(GmGrid* g, uint32_t* counter, uint32_t nblocks, uint32_t flags, uint32_t* seen)
{
    __shared__ uint32_t ok_s, seen_s;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t ok = 1;
        __threadfence();
        uint32_t v = atomicAdd(counter, 1u + flags) + 1u + flags;
        if ((v & 0xFFFFu) != nblocks) {
            const uint64_t deadline = global_ns() + kBarrierWaitNs;
            while (((v = *(volatile uint32_t*)counter) & 0xFFFFu) != nblocks) {
                if (*(volatile int*)&g->error || global_ns() > deadline) {
                    atomicExch(&g->error, 1);
                    ok = 0;
                    break;
                }
            }
        }
        __threadfence();
        ok_s = ok;
        seen_s = v;
    }
    __syncthreads();
    *seen = seen_s;
    return ok_s != 0;
}

// One glutton max search.  GRID = false: one block does everything.  GRID = true:
// every block of a cooperative launch keeps a copy of the level and makes the same
// decisions; the candidate trials of each validity pass are shared out over all
// blocks, results meet in global memory (triple-buffered per pass, one grid barrier per
// pass), and block 0 keeps the global search record.
template <bool GRID>
__global__ void __launch_bounds__(kThreads, 1) gm_kernel(GmLaunch P)
{
    extern __shared__ __align__(16) unsigned char gm_raw[];
    GmSmem& sm = *reinterpret_cast<GmSmem*>(gm_raw);
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t S = P.n, words = (P.n + 7) / 8;
    GmState* st = P.state;
    GmGrid* g = P.grid;
    const bool owner = !GRID || blockIdx.x == 0;
    const uint32_t nblocks = GRID ? gridDim.x : 1u, block = GRID ? blockIdx.x : 0u;
    uint32_t pass_no = 0;  // grid mode: passes so far (selects the exchange buffer)
    bool grid_failed = false;
    // grid mode: rows of a level were stored since the last barrier (every block's share)
    bool stored = false;
    uint32_t extra = 0;    // such barriers so far
    auto load_popped = [&](uint32_t at) {
        if (GRID && stored) {
            // not expected: a fresh level's first pass comes before any pop
            uint32_t seen;
            const uint32_t c = extra % 3;
            if (!grid_sync(g, &g->extra[c], nblocks, 0u, &seen)) grid_failed = true;
            if (block == 0 && tid == 0) g->extra[(c + 2) % 3] = 0;
            ++extra;
            stored = false;
        }
        if (!grid_failed) load_level(sm, P, at, tid);
    };
    for (uint32_t k = tid; k < 256 * 4; k += kThreads) sm.pieces[k >> 2][k & 3] = P.pieces[k];
    for (uint32_t k = tid; k < P.ncolours * 4 * 32; k += kThreads) sm.cc[(k >> 5) & 3u][k >> 7][k & 31u] = P.cc[k];
    uint32_t (*const inval)[32] = reinterpret_cast<uint32_t (*)[32]>(&sm.N[0][0]);  // one-block search
    for (uint32_t k = tid; k < 256; k += kThreads) {
        sm.position_index[k] = st->position_index[k];
        sm.info_index[k] = st->info_index[k];
        sm.played[k] = st->played[k];
        sm.max_played[k] = st->max_played[k];
    }
    if (tid < 8) sm.avail[tid] = st->avail[tid];
    if (tid == 0) {
        sm.level = st->level;
        sm.new_level = st->new_level;
        sm.pop_index = st->pop_index;
        sm.stop = 0;
        sm.trials = st->trials;
        sm.pushes = st->pushes;
        sm.pops = st->pops;
        sm.passes = st->passes;
        sm.levels = st->levels;
        sm.max = st->max;
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
                    else sm.pop_index = pop_state(sm, S);
                    sm.new_level = 0;
                }
                __syncthreads();
                if (sm.level < S) load_popped(sm.level);
                if (grid_failed) break;
                __syncthreads();
                continue;
            }
        }
        if (tid == 0) ++sm.levels;
        // ---- validity fixpoint and scores ----
        bool failed = false;
        for (;;) {
            if (level_statistics(sm, S, nb, P.width, tid)) {
                failed = true;
                break;
            }
            const uint32_t buf = pass_no % 3;
            if (!GRID) {
                for (uint32_t k = tid; k < nb * 32; k += kThreads) inval[k >> 5][k & 31] = 0;
            }
            if (tid == 0) {
                sm.any_invalid = 0;
                sm.trials += sm.sumA;  // every candidate is tried
                ++sm.passes;
            }
            __syncthreads();
            unsigned long long best_key = 0;
            uint32_t best_order = ~0u;
            const bool last_level = level == S - 1;
            const uint32_t c0 = static_cast<uint32_t>(static_cast<uint64_t>(sm.sumA) * block / nblocks);
            const uint32_t c1 = static_cast<uint32_t>(static_cast<uint64_t>(sm.sumA) * (block + 1) / nblocks);
            for (uint32_t from = c0; from < c1; from += kThreads) {
                const uint32_t m = min(c1 - from, static_cast<uint32_t>(kThreads));
                uint32_t log_t = 0;  // threads a trial: as many as there are, at most one a word
                while (log_t < 5 && (m << (log_t + 1)) <= kThreads && (1u << log_t) < words) ++log_t;
                if (((tid & ~31u) >> log_t) >= m) break;  // the whole warp has none
                const uint32_t T = 1u << log_t, sub = tid & (T - 1), c = tid >> log_t;
                const uint32_t order = candidate_of_rank(sm, from + min(c, m - 1));
                uint32_t smallest;
                const unsigned long long key = trial(sm, order, words, T, sub, &smallest);
                if (c >= m) continue;
                if (!smallest) {
                    if (!sub) {
                        const uint32_t i = order >> 10, w = (order >> 5) & 31u;
                        if (GRID) {
                            atomicOr(&g->inval[buf][i][w], 1u << (order & 31u));
                        } else {
                            atomicOr(&inval[i][w], 1u << (order & 31u));
                        }
                        sm.any_invalid = 1;
                    }
                } else if (better_candidate(key, order, best_key, best_order, last_level)) {
                    best_key = key;
                    best_order = order;
                }
            }
            __syncwarp();
            warp_best(best_key, best_order, last_level);
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
                const uint32_t flags = (sm.any_invalid ? kArriveInvalid : 0u) |
                                       (block == 0 && deadline && global_ns() > deadline ? kArriveStop : 0u);
                uint32_t seen;
                if (!grid_sync(g, &g->arrive[buf], nblocks, flags, &seen)) {
                    grid_failed = true;
                    break;
                }
                stored = false;
                // the buffer of the pass before last is free again: every block clears its rows
                const uint32_t old = (pass_no + 2) % 3;
                for (uint32_t j = block + nblocks * warp; j < S; j += nblocks * (kThreads / 32))
                    g->inval[old][j][lane] = 0;
                if (block == 0 && tid == 0) g->arrive[old] = 0;
                const bool any_invalid = (seen & ~kArriveStop) >= kArriveInvalid;
                if (warp == 0 && !any_invalid) {
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
                    if (lane == 0) sm.best_order = o0;
                }
                if (tid == 0) {
                    sm.any_invalid = any_invalid;
                    sm.stop = (seen & kArriveStop) != 0;
                }
                ++pass_no;
            }
            __syncthreads();
            if (!sm.any_invalid) break;
            if (GRID) {
                for (uint32_t k = 4 * tid; k < nb * 32; k += 4 * kThreads) {
                    const uint4 v = __ldcg(reinterpret_cast<const uint4*>(&g->inval[buf][k >> 5][k & 31]));
                    uint32_t* x = &sm.X[k >> 5][k & 31];
                    x[0] &= ~v.x;
                    x[1] &= ~v.y;
                    x[2] &= ~v.z;
                    x[3] &= ~v.w;
                }
            } else {
                for (uint32_t k = tid; k < nb * 32; k += kThreads) sm.X[k >> 5][k & 31] &= ~inval[k >> 5][k & 31];
            }
            __syncthreads();
        }
        if (grid_failed) break;
        if (failed || sm.best_order == ~0u) {
            // remove_invalid_transitions failed or no candidate: pop
            __syncthreads();
            if (tid == 0) {
                if (level == 0) sm.level = ~0u;
                else sm.pop_index = pop_state(sm, S);
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
        if (tid == 0) push_state(sm, S, bi, pos, piece, o);
        __syncthreads();
        if (sm.new_max && tid >= 256 && tid < 256 + sm.max) sm.max_played[tid - 256] = sm.played[tid - 256];
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
                const uint32_t r = sm.X[j][lane] & sm.cc[s2][col - 1][lane];
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
            if (tid == 0) pop_state(sm, S);
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
        st->pushes = sm.pushes;
        st->pops = sm.pops;
        st->passes = sm.passes;
        st->levels = sm.levels;
        st->max = sm.max;
        st->status = grid_failed ? 3 : (level == S ? 0 : (level > S ? 2 : 1));
    }
    if (sm.level < S) store_level(sm, P, sm.level, tid, 0, 1);
    for (uint32_t k = tid; k < 256; k += kThreads) {
        st->position_index[k] = sm.position_index[k];
        st->info_index[k] = sm.info_index[k];
        st->played[k] = sm.played[k];
        st->max_played[k] = sm.max_played[k];
    }
    if (tid < 8) st->avail[tid] = sm.avail[tid];
}

}  // namespace

size_t gm_smem_bytes() { return sizeof(GmSmem); }

cudaError_t launch_gm(const GmLaunch& P, cudaStream_t stream)
{
    const size_t smem = sizeof(GmSmem);
    const void* fn = reinterpret_cast<const void*>(&gm_kernel<false>);
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return e;
    GmLaunch copy = P;
    void* args[] = {&copy};
    return cudaLaunchKernel(fn, dim3(1), dim3(kThreads), args, smem, stream);
}

cudaError_t launch_gm_grid(const GmLaunch& P, uint32_t blocks, cudaStream_t stream)
{
    const size_t smem = sizeof(GmSmem);
    const void* fn = reinterpret_cast<const void*>(&gm_kernel<true>);
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
