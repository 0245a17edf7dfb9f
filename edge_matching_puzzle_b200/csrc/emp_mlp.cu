// Learned value ordering: candidate features, tensor-core inference (tcgen05) and
// f32 training kernels of the scoring network (interface in emp_mlp.h).
#include "emp_mlp.h"

#include <cuda_bf16.h>

#include <algorithm>

namespace emp {

// ---------------------------------------------------------------------------
// feature table (host)

std::vector<uint32_t> build_feature_table(const PuzzleModel& m, const std::vector<LevelPlan>& plan)
{
    const uint32_t n = m.n;
    std::vector<uint32_t> t(kFtCand, 0);
    t[0] = n;
    t[1] = m.width;
    t[2] = m.height;
    t[3] = m.border_id;
    for (uint32_t p = 0; p < n; ++p)
        for (uint32_t s = 0; s < 4; ++s)
            if (m.colours[p][s] < 32) ++t[kFtColours + m.colours[p][s]];
    std::vector<uint32_t> level_of(n, 0);
    for (uint32_t l = 0; l < n; ++l) level_of[plan[l].position] = l;
    for (uint32_t l = 0; l < n; ++l) {
        const uint32_t pos = plan[l].position, x = pos % m.width, y = pos / m.width;
        t[kFtLevelA + l] = pos | (plan[l].kind << 8) | (std::min<uint32_t>(x, 255) << 16) |
                           (std::min<uint32_t>(y, 255) << 24);
        const uint32_t nn = y ? level_of[pos - m.width] : 0xFFFFu;
        const uint32_t ne = x + 1 < m.width ? level_of[pos + 1] : 0xFFFFu;
        const uint32_t ns = y + 1 < m.height ? level_of[pos + m.width] : 0xFFFFu;
        const uint32_t nw = x ? level_of[pos - 1] : 0xFFFFu;
        t[kFtLevelB + 2 * l] = nn | (ne << 16);
        t[kFtLevelB + 2 * l + 1] = ns | (nw << 16);
    }
    uint32_t off = kFtCand;
    for (uint32_t k = 0; k < 3; ++k) {
        t[kFtKindOff + k] = off;
        off += 4 * m.nb_kind(k);
    }
    t.resize(off, 0);
    for (uint32_t k = 0; k < 3; ++k)
        for (uint32_t e = 0; e < 4 * m.nb_kind(k); ++e) {
            const uint32_t p = m.members[k][e >> 2], o = e & 3u;
            uint32_t col = 0;
            for (uint32_t s = 0; s < 4; ++s) col |= (m.colour(p, s, o) & 31u) << (5 * s);
            t[t[kFtKindOff + k] + e] = (p << 20) | col;
        }
    while (t.size() % 4) t.push_back(0);  // tables concatenate 16-byte aligned
    return t;
}

namespace {

constexpr unsigned kFull = 0xFFFFFFFFu;

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ uint32_t side_colour(uint32_t cand, uint32_t s) { return (cand >> (5 * s)) & 31u; }

__device__ __forceinline__ uint32_t colour_edges(uint32_t cand, uint32_t c)
{
    return (side_colour(cand, 0) == c) + (side_colour(cand, 1) == c) + (side_colour(cand, 2) == c) +
           (side_colour(cand, 3) == c);
}

// ---------------------------------------------------------------------------
// features: a warp takes eight rows and clears them, then four lanes a row count the colours of the
// placed pieces and the first of them sets the active entries.  bf16 rows go straight into the
// operand images of the inference (below), in which eight rows are whole lines.
//
//   [0, 128)    colour of each side of the oriented candidate (4 x 32 one-hot)
//   [128, 140)  state of each side's neighbour: outside / placed / free (4 x 3)
//   [140, 204)  free sides: edges of that colour still on unplaced pieces, 0..15+ (4 x 16)
//   [204, 236)  x and y of the position (2 x 16)
//   [236, 252)  depth: level * 16 / n
//   [252, 255)  kind: centre / border / corner
//   255         constant 1
//   [256, 512)  colours of the first two free sides, hashed (c1 * 32 + c2) mod 256
// Operand images of the inference: row r of a tile of `rows` rows, element k, in chunks of
// kKc elements of K, each in the canonical K-major layout without swizzle: 8-row x 16-byte core
// matrices, K-adjacent ones 128 bytes apart, 8-row groups kKc * 16 bytes apart.
constexpr uint32_t kKc = 64, kTileRows = 128;
__device__ __forceinline__ uint32_t image_offset(uint32_t r, uint32_t k, uint32_t rows)
{
    return (k / kKc) * (rows * kKc * 2) + (r >> 3) * (kKc * 16) + ((k % kKc) >> 3) * 128 + (r & 7u) * 16 + (k & 7u) * 2;
}
constexpr uint32_t kXTileBytes = kTileRows * kMlpIn * 2;

__global__ void features_kernel(const uint32_t* __restrict__ ftab, const unsigned long long* __restrict__ ftab_off,
                                const FeatItem* __restrict__ items, uint64_t n, const uint16_t* __restrict__ prefixes,
                                uint8_t* __restrict__ image, float* __restrict__ out_f32)
{
    const uint32_t lane = threadIdx.x & 31u, sub = lane & 3u;
    const uint64_t nwarps = (static_cast<uint64_t>(gridDim.x) * blockDim.x) >> 5;
    for (uint64_t g = (blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x) >> 5; g * 8 < n; g += nwarps) {
        if (image) {
            // the group's 1 KB in each chunk (rows past n belong to the last tile and are cleared too)
            uint8_t* tile = image + (g / (kTileRows / 8)) * kXTileBytes;
            const uint32_t off = static_cast<uint32_t>(g % (kTileRows / 8)) * (kKc * 16);
            for (uint32_t c = 0; c < kMlpIn / kKc; ++c) {
                uint4* q = reinterpret_cast<uint4*>(tile + c * (kTileRows * kKc * 2) + off);
                q[lane] = make_uint4(0, 0, 0, 0);
                q[lane + 32] = make_uint4(0, 0, 0, 0);
            }
        } else {
            for (uint64_t r = g * 8; r < g * 8 + 8 && r < n; ++r) {
                uint4* row = reinterpret_cast<uint4*>(out_f32 + r * kMlpIn);
                for (uint32_t j = 0; j < 4; ++j) row[lane + 32 * j] = make_uint4(0, 0, 0, 0);
            }
        }
        __syncwarp();
        const bool mine = g * 8 + (lane >> 2) < n;
        const uint64_t i = mine ? g * 8 + (lane >> 2) : n - 1;
        const FeatItem it = items[i];
        const uint32_t* T = ftab + ftab_off[it.puzzle];
        const uint32_t l = it.len, nlev = T[0];
        const uint32_t A = T[kFtLevelA + l];
        const uint32_t kind = (A >> 8) & 0xFFu;
        const uint32_t x = min((A >> 16) & 0xFFu, 15u), y = min(A >> 24, 15u);
        const uint32_t cand = T[T[kFtKindOff + kind] + it.t];
        const uint32_t b0 = T[kFtLevelB + 2 * l], b1 = T[kFtLevelB + 2 * l + 1];
        const uint32_t nb[4] = {b0 & 0xFFFFu, b0 >> 16, b1 & 0xFFFFu, b1 >> 16};
        // edges of each free side's colour on the pieces placed before this level
        const uint16_t* pre = prefixes + it.prefix_off;
        uint32_t placed[4] = {0, 0, 0, 0};
        for (uint32_t j = sub; j < l; j += 4) {
            const uint32_t kj = (T[kFtLevelA + j] >> 8) & 0xFFu;
            const uint32_t cj = T[T[kFtKindOff + kj] + pre[j]];
            for (uint32_t s = 0; s < 4; ++s) placed[s] += colour_edges(cj, side_colour(cand, s));
        }
        __syncwarp();
        for (uint32_t s = 0; s < 4; ++s) {
            placed[s] += __shfl_xor_sync(kFull, placed[s], 1);
            placed[s] += __shfl_xor_sync(kFull, placed[s], 2);
        }
        if (mine && sub == 0) {
            uint8_t* tile = image + (i / kTileRows) * kXTileBytes;
            const uint32_t r = static_cast<uint32_t>(i % kTileRows);
            auto set = [&](uint32_t k) {
                if (image) *reinterpret_cast<uint16_t*>(tile + image_offset(r, k, kTileRows)) = 0x3F80u;  // bf16 1.0
                else out_f32[i * kMlpIn + k] = 1.0f;
            };
            uint32_t free0 = 0, free1 = 0, nfree = 0;
#pragma unroll
            for (uint32_t s = 0; s < 4; ++s) {
                const uint32_t c = side_colour(cand, s);
                set(32 * s + c);
                const uint32_t state = nb[s] == 0xFFFFu ? 0u : (nb[s] < l ? 1u : 2u);
                set(128 + 3 * s + state);
                if (state == 2) {
                    const uint32_t left = T[kFtColours + c] - placed[s] - colour_edges(cand, c);
                    set(140 + 16 * s + min(left, 15u));
                    if (nfree == 0) free0 = c;
                    if (nfree == 1) free1 = c;
                    ++nfree;
                }
            }
            set(204 + x);
            set(220 + y);
            set(236 + min(l * 16 / max(nlev, 1u), 15u));
            set(252 + min(kind, 2u));
            set(255);
            if (nfree >= 2) set(256 + ((free0 * 32 + free1) & 255u));
            else if (nfree == 1) set(256 + free0);
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// tensor-core inference
//
// One persistent CTA an SM scores 128 rows at a time:
//   layer 1  D1[128 x 256] = X[128 x 512] . W1^T      8 chunks of K = 64
//   layer 2  D2[128 x 256] = relu(D1 + b1) . W2^T     4 chunks of K = 64
//   score    relu(D2 + b2) . w3 + b3                  in the epilogue
// X, W1 and W2 lie in memory as operand images (image_offset), so a chunk is one or two bulk copies
// into one of three stages.  One thread issues the copies, one the MMAs, and four warps read the
// accumulators (tensor memory: D1 in columns [0, 256), D2 in [256, 512)), so that the copies run
// ahead and the score of a tile overlaps layer 1 of the next.  tcgen05.commit frees stages and
// reports accumulators.
//
// What bounds it: the copies on their way.  160 000 rows take 74 us, 14 000 cycles a tile: 512 KB
// (384 KB of weights) arrive at 37 bytes a cycle in an SM while the tensor pipe is active 44 % of the
// time, and L2 (27 %) and DRAM (28 %) have room.  Measured on a B200, before (one warpgroup that staged chunks with plain loads
// and waited for each) and after: 353 000 rows, 65 536 a launch, 2.04 ms -> 0.21 ms; a whole call
// scoring 19 rows 107 us -> 81 us.
constexpr uint32_t kStages = 3;
constexpr uint32_t kXBytes = kTileRows * kKc * 2, kWBytes = kMlpHidden * kKc * 2;  // a chunk: 16 KB, 32 KB
constexpr uint32_t kSmW = kXBytes, kStageBytes = kXBytes + kWBytes;
constexpr uint32_t kSmH = kStages * kStageBytes;          // 128 x 256 bf16: 64 KB
constexpr uint32_t kSmVec = kSmH + kTileRows * kMlpHidden * 2;  // b1, b2, w3 (f32)
constexpr uint32_t kSmBar = kSmVec + 3 * kMlpHidden * 4;
enum : uint32_t { kBarFull = 0, kBarEmpty = kStages, kBarD1 = 2 * kStages, kBarH, kBarD2, kBarD2Free, kBarDrain, kBars };
constexpr uint32_t kSmSlot = kSmBar + 8 * kBars;
constexpr uint32_t kSmTotal = kSmSlot + 16;
constexpr unsigned long long kWaitNs = 2000000000ull;     // 2 s per wait
constexpr uint32_t kInferThreads = 192;                   // 4 epilogue warps, copies, MMAs

// byte offset of element (r, k) in a K-major canonical tile whose rows hold kk elements
__device__ __forceinline__ uint32_t canon(uint32_t r, uint32_t k, uint32_t kk)
{
    return (r >> 3) * (kk * 16) + (k >> 3) * 128 + (r & 7u) * 16 + (k & 7u) * 2;
}

__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo)
{
    uint64_t d = 0;
    d |= static_cast<uint64_t>((addr >> 4) & 0x3FFFu);
    d |= static_cast<uint64_t>((lbo >> 4) & 0x3FFFu) << 16;
    d |= static_cast<uint64_t>((sbo >> 4) & 0x3FFFu) << 32;
    d |= 1ull << 46;  // descriptor version of sm_100
    return d;         // base offset 0, layout type 0 (no swizzle)
}

// kind::f16 instruction descriptor: F32 accumulate, BF16 A and B, both K-major,
// N = 256, M = 128
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((kMlpHidden >> 3) << 17) | ((kTileRows >> 4) << 24);

__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t accumulate)
{
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(kIdesc), "r"(accumulate));
}

__device__ __forceinline__ void mma_commit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity)
{
    const unsigned long long deadline = global_ns() + kWaitNs;
    for (;;) {
        uint32_t done;
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
        if (global_ns() > deadline) return false;
    }
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// 32 consecutive f32 accumulator columns of this thread's row
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float* v)
{
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
}

__device__ __forceinline__ void bar_init(uint32_t bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void bar_expect(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

__global__ void __launch_bounds__(kInferThreads, 1)
    mlp_infer_kernel(const uint8_t* __restrict__ x, uint64_t n, const uint8_t* __restrict__ w1,
                     const uint8_t* __restrict__ w2, const float* __restrict__ params, float* __restrict__ out,
                     int* err)
{
    extern __shared__ __align__(1024) uint8_t sm[];
    const uint32_t tid = threadIdx.x, warp = tid >> 5;
    const uint32_t base = static_cast<uint32_t>(__cvta_generic_to_shared(sm));
    auto bar = [&](uint32_t k) { return base + kSmBar + 8 * k; };
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + kSmSlot);
    float* vb1 = reinterpret_cast<float*>(sm + kSmVec);
    float* vb2 = vb1 + kMlpHidden;
    float* vw3 = vb2 + kMlpHidden;
    for (uint32_t j = tid; j < kMlpHidden; j += kInferThreads) {
        vb1[j] = params[kOffB1 + j];
        vb2[j] = params[kOffB2 + j];
        vw3[j] = params[kOffW3 + j];
    }
    const float b3 = params[kOffB3];
    if (tid == 0) {
        for (uint32_t k = 0; k < kBars; ++k) bar_init(bar(k), k == kBarH || k == kBarD2Free ? 128u : 1u);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        const uint32_t slot = static_cast<uint32_t>(__cvta_generic_to_shared(tmem_slot));
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(slot) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tmem_slot;
    const uint32_t d1 = tmem, d2 = tmem + kMlpHidden;
    const uint64_t tiles = (n + kTileRows - 1) / kTileRows;
    constexpr uint32_t kC1 = kMlpIn / kKc, kC2 = kMlpHidden / kKc;
    bool ok = true;
    uint32_t issued = 0;  // copy thread: chunks whose copies were issued

    if (warp == 4 && (tid & 31u) == 0) {
        // ---- copies: a tile's chunks of X and W1, then of W2 ----
        for (uint64_t tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
            for (uint32_t c = 0; c < kC1 + kC2 && ok; ++c) {
                const uint32_t s = issued % kStages;
                ok = bar_wait(bar(kBarEmpty + s), ((issued / kStages) & 1u) ^ 1u);
                if (!ok) break;
                const uint32_t dst = base + s * kStageBytes, full = bar(kBarFull + s);
                if (c < kC1) {
                    bar_expect(full, kXBytes + kWBytes);
                    bulk_copy(dst, x + tile * kXTileBytes + c * kXBytes, kXBytes, full);
                    bulk_copy(dst + kSmW, w1 + c * kWBytes, kWBytes, full);
                } else {
                    bar_expect(full, kWBytes);
                    bulk_copy(dst + kSmW, w2 + (c - kC1) * kWBytes, kWBytes, full);
                }
                ++issued;
            }
        }
        // copies in flight have landed before the CTA's shared memory goes away
        for (uint32_t k = issued > kStages ? issued - kStages : 0; k < issued; ++k)
            bar_wait(bar(kBarFull + k % kStages), (k / kStages) & 1u);
    } else if (warp == 5 && (tid & 31u) == 0) {
        // ---- MMAs ----
        uint32_t k = 0, t = 0;  // chunks and tiles so far
        for (uint64_t tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x, ++t) {
            // D1 is free: the epilogue has read it when it hands over H
            if (t) ok = bar_wait(bar(kBarH), (t - 1) & 1u);
            for (uint32_t c = 0; c < kC1 + kC2 && ok; ++c, ++k) {
                if (c == kC1) {
                    mma_commit(bar(kBarD1));
                    ok = bar_wait(bar(kBarH), t & 1u);  // relu(D1 + b1) is in shared memory
                    if (ok && t) ok = bar_wait(bar(kBarD2Free), (t - 1) & 1u);
                    if (!ok) break;
                }
                const uint32_t s = k % kStages;
                ok = bar_wait(bar(kBarFull + s), (k / kStages) & 1u);
                if (!ok) break;
                fence_after();
                const uint32_t at = base + s * kStageBytes;
                for (uint32_t kk = 0; kk < kKc / 16; ++kk) {
                    const uint64_t b = smem_desc(at + kSmW + kk * 256, 128, kKc * 16);
                    if (c < kC1)
                        mma_bf16(d1, smem_desc(at + kk * 256, 128, kKc * 16), b, (c | kk) != 0);
                    else
                        mma_bf16(d2, smem_desc(base + kSmH + ((c - kC1) * (kKc / 8) + kk * 2) * 128, 128, kMlpHidden * 16),
                                 b, ((c - kC1) | kk) != 0);
                }
                mma_commit(bar(kBarEmpty + s));
            }
            if (ok) mma_commit(bar(kBarD2));
        }
        // MMAs in flight have ended before tensor memory is freed
        mma_commit(bar(kBarDrain));
        bar_wait(bar(kBarDrain), 0);
    } else if (warp < 4) {
        // ---- epilogues: this thread's row is its tensor-memory lane ----
        const uint32_t lane_base = (32u * warp) << 16, r = tid;
        uint32_t t = 0;
        for (uint64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++t) {
            ok = bar_wait(bar(kBarD1), t & 1u);
            if (!__all_sync(kFull, ok)) break;
            fence_after();
            // bias, relu, bf16 into the layer-2 operand (layer 2 of the tile before has ended: its score
            // was taken)
            for (uint32_t c0 = 0; c0 < kMlpHidden; c0 += 32) {
                float v[32];
                tmem_ld32(d1 + lane_base + c0, v);
                for (uint32_t g = 0; g < 4; ++g) {
                    uint32_t w[4];
                    for (uint32_t h = 0; h < 4; ++h) {
                        const uint32_t j = c0 + g * 8 + 2 * h;
                        const __nv_bfloat162 pr = __floats2bfloat162_rn(fmaxf(v[g * 8 + 2 * h] + vb1[j], 0.f),
                                                                        fmaxf(v[g * 8 + 2 * h + 1] + vb1[j + 1], 0.f));
                        w[h] = *reinterpret_cast<const uint32_t*>(&pr);
                    }
                    *reinterpret_cast<uint4*>(sm + kSmH + canon(r, c0 + g * 8, kMlpHidden)) =
                        make_uint4(w[0], w[1], w[2], w[3]);
                }
            }
            fence_proxy_async();
            fence_before();
            bar_arrive(bar(kBarH));
            ok = bar_wait(bar(kBarD2), t & 1u);
            if (!__all_sync(kFull, ok)) break;
            fence_after();
            // bias, relu, dot with w3
            float score = b3;
            for (uint32_t c0 = 0; c0 < kMlpHidden; c0 += 32) {
                float v[32];
                tmem_ld32(d2 + lane_base + c0, v);
#pragma unroll
                for (int j = 0; j < 32; ++j) score += fmaxf(v[j] + vb2[c0 + j], 0.f) * vw3[c0 + j];
            }
            fence_before();
            bar_arrive(bar(kBarD2Free));
            const uint64_t row = tile * kTileRows + r;
            if (row < n) out[row] = score;
        }
    }
    if (!ok) atomicExch(err, 1);
    __syncwarp();
    fence_before();
    __syncthreads();
    if (warp == 0) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
    }
}

// ---------------------------------------------------------------------------
// f32 training kernels

// C(m, n) = sum_k A(m, k) B(k, n) in 64x64 tiles of 256 threads, 4x4 outputs a thread, 16 k a step,
// the next step's operands on their way in registers while this one is multiplied.
//   TA: A(m, k) = A[k * lda + m], else A[m * lda + k];  TB: B(k, n) = B[n * ldb + k], else B[k * ldb + n]
// N is a multiple of 64.  Without TA, K is a multiple of 16 and M any; with TA (sums over rows) M is
// a multiple of 64 and K any, and blockIdx.z takes k in [z * kchunk, (z + 1) * kchunk) into the z-th of
// gridDim.z partial results: a 256x256 gradient has 16 tiles, which alone leave most SMs idle.
// Measured on a B200 at 2048 rows, before (32x32 tiles, an element a load, no split) and after:
// layer 1 forward 96 us and bias 4 us -> 37 us (128 blocks of 8 warps: latency), its weight
// gradient 179 us -> 21 us, a whole loss and gradient 0.95 ms -> 0.14 ms; the gradient's error
// against 64 bits 4e-7 .. 1e-6 -> 8e-8, for the sums are shorter.
constexpr int kTile = kMlpTile, kTk = 16, kTs = kTile + 4;

enum class Epilogue {
    kBiasRelu,  // C = max(v + bias[n], 0)
    kMask,      // C = gate[m][n] > 0 ? v : 0, and the tile's column sums of C into sums[blockIdx.y][n]
    kPartial,   // C[blockIdx.z] = v
};

template <bool TA, bool TB, Epilogue E>
__global__ void __launch_bounds__(256) gemm_f32_kernel(const float* __restrict__ A, uint32_t lda,
                                                       const float* __restrict__ B, uint32_t ldb, float* __restrict__ C,
                                                       uint32_t M, uint32_t N, uint32_t K, uint32_t kchunk,
                                                       const float* __restrict__ bias, const float* __restrict__ gate,
                                                       float* __restrict__ sums)
{
    __shared__ __align__(16) float As[2][kTk][kTs];
    __shared__ __align__(16) float Bs[2][kTk][kTs];
    const uint32_t tid = threadIdx.x, tx = tid & 15u, ty = tid >> 4;
    const uint32_t m0 = blockIdx.y * kTile, n0 = blockIdx.x * kTile;
    const uint32_t kbegin = blockIdx.z * kchunk, kend = min(K, kbegin + kchunk);
    float4 ra, rb;
    // operand steps: 4 consecutive elements a thread
    auto fetch = [&](uint32_t k0) {
        if (TA) {
            const uint32_t k = k0 + (tid >> 4);
            ra = k < kend ? *reinterpret_cast<const float4*>(A + static_cast<uint64_t>(k) * lda + m0 + 4 * (tid & 15u))
                          : make_float4(0.f, 0.f, 0.f, 0.f);
        } else {
            const uint32_t m = m0 + (tid >> 2);
            ra = m < M ? *reinterpret_cast<const float4*>(A + static_cast<uint64_t>(m) * lda + k0 + 4 * (tid & 3u))
                       : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if (TB) {
            const uint32_t n = n0 + (tid >> 2);
            rb = *reinterpret_cast<const float4*>(B + static_cast<uint64_t>(n) * ldb + k0 + 4 * (tid & 3u));
        } else {
            const uint32_t k = k0 + (tid >> 4);
            rb = k < kend ? *reinterpret_cast<const float4*>(B + static_cast<uint64_t>(k) * ldb + n0 + 4 * (tid & 15u))
                          : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    auto store = [&](int buf) {
        if (TA) {
            *reinterpret_cast<float4*>(&As[buf][tid >> 4][4 * (tid & 15u)]) = ra;
        } else {
            const uint32_t k = 4 * (tid & 3u), m = tid >> 2;
            As[buf][k][m] = ra.x;
            As[buf][k + 1][m] = ra.y;
            As[buf][k + 2][m] = ra.z;
            As[buf][k + 3][m] = ra.w;
        }
        if (TB) {
            const uint32_t k = 4 * (tid & 3u), n = tid >> 2;
            Bs[buf][k][n] = rb.x;
            Bs[buf][k + 1][n] = rb.y;
            Bs[buf][k + 2][n] = rb.z;
            Bs[buf][k + 3][n] = rb.w;
        } else {
            *reinterpret_cast<float4*>(&Bs[buf][tid >> 4][4 * (tid & 15u)]) = rb;
        }
    };
    float acc[4][4] = {};
    int buf = 0;
    if (kbegin < kend) {
        fetch(kbegin);
        store(0);
    }
    __syncthreads();
    for (uint32_t k0 = kbegin; k0 < kend; k0 += kTk) {
        const bool more = k0 + kTk < kend;
        if (more) fetch(k0 + kTk);
#pragma unroll
        for (int k = 0; k < kTk; ++k) {
            const float4 a = *reinterpret_cast<const float4*>(&As[buf][k][4 * ty]);
            const float4 b = *reinterpret_cast<const float4*>(&Bs[buf][k][4 * tx]);
            const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] += av[i] * bv[j];
        }
        if (more) store(buf ^ 1);
        __syncthreads();
        buf ^= 1;
    }
    const uint32_t n = n0 + 4 * tx;
    float col[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t m = m0 + 4 * ty + i;
        if (m >= M) continue;
        float4 v = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        float* c = C + (E == Epilogue::kPartial ? static_cast<uint64_t>(blockIdx.z) * M * N : 0ull) +
                   static_cast<uint64_t>(m) * N + n;
        if (E == Epilogue::kBiasRelu) {
            v.x = fmaxf(v.x + bias[n], 0.f);
            v.y = fmaxf(v.y + bias[n + 1], 0.f);
            v.z = fmaxf(v.z + bias[n + 2], 0.f);
            v.w = fmaxf(v.w + bias[n + 3], 0.f);
        }
        if (E == Epilogue::kMask) {
            const float4 h = *reinterpret_cast<const float4*>(gate + static_cast<uint64_t>(m) * N + n);
            v.x = h.x > 0.f ? v.x : 0.f;
            v.y = h.y > 0.f ? v.y : 0.f;
            v.z = h.z > 0.f ? v.z : 0.f;
            v.w = h.w > 0.f ? v.w : 0.f;
            col[0] += v.x;
            col[1] += v.y;
            col[2] += v.z;
            col[3] += v.w;
        }
        *reinterpret_cast<float4*>(c) = v;
    }
    if (E == Epilogue::kMask) {
        float (*const red)[kTs] = As[0];  // 16 rows, one per ty
        *reinterpret_cast<float4*>(&red[ty][4 * tx]) = make_float4(col[0], col[1], col[2], col[3]);
        __syncthreads();
        if (tid < kTile) {
            float v = 0.f;
            for (int r = 0; r < 16; ++r) v += red[r][tid];
            sums[static_cast<uint64_t>(blockIdx.y) * N + n0 + tid] = v;
        }
    }
}

// s[r] = h2[r] . w3 + b3 (one warp per row)
__global__ void score_f32_kernel(const float* __restrict__ h2, const float* __restrict__ params, uint64_t rows,
                                 float* __restrict__ s)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t nw = (static_cast<uint64_t>(gridDim.x) * blockDim.x) >> 5;
    for (uint64_t r = (blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x) >> 5; r < rows; r += nw) {
        float acc = 0.f;
        for (uint32_t j = lane; j < kMlpHidden; j += 32) acc += h2[r * kMlpHidden + j] * params[kOffW3 + j];
        for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(kFull, acc, o);
        if (lane == 0) s[r] = acc + params[kOffB3];
    }
}

// weighted logistic loss: loss[0] += w * (softplus(s) - y s), loss[1] += w; ds = w (sigmoid(s) - y)
__global__ void loss_kernel(const float* __restrict__ s, const float* __restrict__ y, const float* __restrict__ wt,
                            uint64_t rows, float* __restrict__ ds, double* loss)
{
    double l = 0, wsum = 0;
    for (uint64_t r = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; r < rows;
         r += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const float v = s[r], w = wt[r];
        const float sp = v > 0.f ? v + log1pf(expf(-v)) : log1pf(expf(v));
        const float sig = 1.f / (1.f + expf(-v));
        l += static_cast<double>(w) * (sp - y[r] * v);
        wsum += w;
        ds[r] = w * (sig - y[r]);
    }
    for (int o = 16; o; o >>= 1) {
        l += __shfl_xor_sync(kFull, l, o);
        wsum += __shfl_xor_sync(kFull, wsum, o);
    }
    if ((threadIdx.x & 31u) == 0) {
        atomicAdd(&loss[0], l);
        atomicAdd(&loss[1], wsum);
    }
}

// Rows of 32, a thread a column: d = ds / sum of weights; dh2 = d (x) w3 where h2 > 0, and the partial
// sums of dw3 = h2^T d, db2 = column sums of dh2 and db3 = sum of d, [block][2 * kMlpHidden + 1].
constexpr uint32_t kColRows = kMlpColRows, kColParts = kMlpColParts;

__global__ void __launch_bounds__(kMlpHidden)
    backward_columns_kernel(const float* __restrict__ ds, const float* __restrict__ h2, const float* __restrict__ params,
                            const double* __restrict__ loss, uint64_t rows, float* __restrict__ dh2,
                            float* __restrict__ parts)
{
    __shared__ float d[kColRows];
    const uint32_t j = threadIdx.x;
    const uint64_t r0 = static_cast<uint64_t>(blockIdx.x) * kColRows;
    const uint32_t count = static_cast<uint32_t>(rows - r0 < kColRows ? rows - r0 : kColRows);
    const float inv = loss[1] > 0 ? static_cast<float>(1.0 / loss[1]) : 0.f;
    if (j < kColRows) d[j] = j < count ? ds[r0 + j] * inv : 0.f;
    __syncthreads();
    const float w3 = params[kOffW3 + j];
    float dw3 = 0.f, db2 = 0.f;
    for (uint32_t r = 0; r < count; ++r) {
        const float h = h2[(r0 + r) * kMlpHidden + j];
        const float v = h > 0.f ? d[r] * w3 : 0.f;
        dh2[(r0 + r) * kMlpHidden + j] = v;
        dw3 += d[r] * h;
        db2 += v;
    }
    float* p = parts + static_cast<uint64_t>(blockIdx.x) * kColParts;
    p[j] = dw3;
    p[kMlpHidden + j] = db2;
    if (j < 32) {
        float v = d[j];
        for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
        if (j == 0) p[2 * kMlpHidden] = v;
    }
}

// every parameter's gradient from its partial sums, added in order
__global__ void reduce_gradient_kernel(const float* __restrict__ pw1, uint32_t z1, const float* __restrict__ pw2,
                                       uint32_t z2, const float* __restrict__ pb1, uint32_t row_tiles,
                                       const float* __restrict__ pcol, uint32_t col_blocks, float* __restrict__ grad)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kMlpParams) return;
    const float* p;
    uint32_t count, stride;
    if (i < kOffB1) {
        p = pw1 + i;
        count = z1;
        stride = kMlpHidden * kMlpIn;
    } else if (i < kOffW2) {
        p = pb1 + (i - kOffB1);
        count = row_tiles;
        stride = kMlpHidden;
    } else if (i < kOffB2) {
        p = pw2 + (i - kOffW2);
        count = z2;
        stride = kMlpHidden * kMlpHidden;
    } else {
        // parts hold dw3, db2, db3
        p = pcol + (i < kOffW3 ? kMlpHidden + (i - kOffB2) : i < kOffB3 ? i - kOffW3 : 2 * kMlpHidden);
        count = col_blocks;
        stride = kColParts;
    }
    float v = 0.f;
    for (uint32_t k = 0; k < count; ++k) v += p[static_cast<uint64_t>(k) * stride];
    grad[i] = v;
}

__global__ void adam_kernel(float* p, const float* __restrict__ g, float* m1, float* m2, uint32_t n, float lr,
                            float c1, float c2)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float a = 0.9f * m1[i] + 0.1f * gi;
        const float b = 0.999f * m2[i] + 0.001f * gi * gi;
        m1[i] = a;
        m2[i] = b;
        p[i] -= lr * (a / c1) / (sqrtf(b / c2) + 1e-8f);
    }
}

// a weight matrix (rows x cols, row-major) into its operand image
__global__ void pack_bf16_kernel(const float* __restrict__ src, uint8_t* __restrict__ dst, uint32_t rows, uint32_t cols)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < rows * cols; i += gridDim.x * blockDim.x)
        *reinterpret_cast<__nv_bfloat16*>(dst + image_offset(i / cols, i % cols, rows)) = __float2bfloat16_rn(src[i]);
}

uint32_t grid_for(uint64_t n, uint32_t threads)
{
    return static_cast<uint32_t>(std::min<uint64_t>((n + threads - 1) / threads, 148ull * 16));
}

// f32 feature rows into operand images; eight lanes write one line of eight rows' 16 bytes
__global__ void rows_to_image_kernel(const float* __restrict__ src, uint8_t* __restrict__ image, uint64_t n)
{
    constexpr uint32_t kPieces = kMlpIn / 8;
    const uint64_t total = (n + 7) / 8 * 8 * kPieces;
    for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const uint64_t row = i / (8 * kPieces) * 8 + (i & 7u);
        const uint32_t k = static_cast<uint32_t>(i / 8 % kPieces) * 8;
        if (row >= n) continue;
        const float4 a = *reinterpret_cast<const float4*>(src + row * kMlpIn + k);
        const float4 b = *reinterpret_cast<const float4*>(src + row * kMlpIn + k + 4);
        const __nv_bfloat162 p[4] = {__floats2bfloat162_rn(a.x, a.y), __floats2bfloat162_rn(a.z, a.w),
                                     __floats2bfloat162_rn(b.x, b.y), __floats2bfloat162_rn(b.z, b.w)};
        *reinterpret_cast<uint4*>(image + (row / kTileRows) * kXTileBytes +
                                  image_offset(static_cast<uint32_t>(row % kTileRows), k, kTileRows)) =
            *reinterpret_cast<const uint4*>(p);
    }
}

__global__ void gather_rows_kernel(const float* __restrict__ src, const uint32_t* __restrict__ idx, uint64_t n,
                                   uint32_t cols, float* __restrict__ dst, const float* __restrict__ y,
                                   const float* __restrict__ w, float* __restrict__ y_out, float* __restrict__ w_out)
{
    for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n * cols;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const uint64_t r = i / cols;
        const uint32_t c = static_cast<uint32_t>(i % cols);
        const uint64_t from = idx[r];
        dst[i] = src[from * cols + c];
        if (c == 0) {
            y_out[r] = y[from];
            w_out[r] = w[from];
        }
    }
}

// item (prefix first + j, level 1 + k); levels at or past the puzzle's own prefix
// length get len = 0 (skipped when summing)
__global__ void order_items_kernel(const uint16_t* __restrict__ prefixes, const uint32_t* __restrict__ prefix_puzzle,
                                   const uint32_t* __restrict__ puzzle_depth, uint32_t depth, uint64_t first,
                                   uint64_t count, FeatItem* __restrict__ items)
{
    const uint32_t per = depth - 1;
    for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < count * per;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const uint64_t p = first + i / per;
        const uint32_t l = 1 + static_cast<uint32_t>(i % per);
        const uint32_t pz = prefix_puzzle[p];
        const uint32_t len = puzzle_depth ? puzzle_depth[pz] : depth;
        FeatItem it;
        it.prefix_off = p * depth;
        it.puzzle = pz;
        if (l < len) {
            it.len = static_cast<uint16_t>(l);
            it.t = prefixes[p * depth + l];
        } else {
            it.len = 0;
            it.t = prefixes[p * depth];
        }
        items[i] = it;
    }
}

__global__ void order_accumulate_kernel(const float* __restrict__ scores, const FeatItem* __restrict__ items,
                                        uint64_t count, uint32_t depth, float* __restrict__ prefix_score)
{
    const uint32_t per = depth - 1;
    for (uint64_t j = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; j < count;
         j += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        float acc = 0.f;
        for (uint32_t k = 0; k < per; ++k) {
            const uint64_t i = j * per + k;
            if (!items[i].len) continue;
            const float v = scores[i];
            acc -= fmaxf(-v, 0.f) + log1pf(expf(-fabsf(v)));  // log sigmoid(v)
        }
        prefix_score[j] = acc;
    }
}

}  // namespace

uint64_t mlp_image_bytes(uint64_t n) { return (n + kTileRows - 1) / kTileRows * kXTileBytes; }

cudaError_t launch_rows_to_image(const float* src, void* image, uint64_t n, cudaStream_t stream)
{
    if (!n) return cudaSuccess;
    rows_to_image_kernel<<<grid_for((n + 7) / 8 * 8 * (kMlpIn / 8), 256), 256, 0, stream>>>(
        src, static_cast<uint8_t*>(image), n);
    return cudaGetLastError();
}

cudaError_t launch_gather_rows(const float* src, const uint32_t* idx, uint64_t n, uint32_t cols, float* dst,
                               const float* y, const float* w, float* y_out, float* w_out, cudaStream_t stream)
{
    if (!n) return cudaSuccess;
    gather_rows_kernel<<<grid_for(n * cols, 256), 256, 0, stream>>>(src, idx, n, cols, dst, y, w, y_out, w_out);
    return cudaGetLastError();
}

cudaError_t launch_order_items(const uint16_t* prefixes, const uint32_t* prefix_puzzle, const uint32_t* puzzle_depth,
                               uint32_t depth, uint64_t first, uint64_t count, FeatItem* items, cudaStream_t stream)
{
    if (!count || depth < 2) return cudaSuccess;
    order_items_kernel<<<grid_for(count * (depth - 1), 256), 256, 0, stream>>>(prefixes, prefix_puzzle, puzzle_depth,
                                                                               depth, first, count, items);
    return cudaGetLastError();
}

cudaError_t launch_order_accumulate(const float* scores, const FeatItem* items, uint64_t count, uint32_t depth,
                                    float* prefix_score, cudaStream_t stream)
{
    if (!count || depth < 2) return cudaSuccess;
    order_accumulate_kernel<<<grid_for(count, 256), 256, 0, stream>>>(scores, items, count, depth, prefix_score);
    return cudaGetLastError();
}

cudaError_t launch_features(const uint32_t* ftab, const unsigned long long* ftab_off, const FeatItem* items,
                            uint64_t n, const uint16_t* prefixes, void* image, float* out_f32, cudaStream_t stream)
{
    if (!n) return cudaSuccess;
    const uint64_t blocks = std::min<uint64_t>((n + 31) / 32, 148ull * 64);  // 4 warps of eight rows
    features_kernel<<<static_cast<uint32_t>(blocks), 128, 0, stream>>>(
        ftab, ftab_off, items, n, prefixes, static_cast<uint8_t*>(image), out_f32);
    return cudaGetLastError();
}

cudaError_t launch_mlp_pack_bf16(const MlpDevice& m, cudaStream_t stream)
{
    pack_bf16_kernel<<<256, 256, 0, stream>>>(m.params + kOffW1, reinterpret_cast<uint8_t*>(m.w1_bf16), kMlpHidden,
                                              kMlpIn);
    pack_bf16_kernel<<<256, 256, 0, stream>>>(m.params + kOffW2, reinterpret_cast<uint8_t*>(m.w2_bf16), kMlpHidden,
                                              kMlpHidden);
    return cudaGetLastError();
}

size_t mlp_infer_smem_bytes() { return kSmTotal; }

cudaError_t launch_mlp_infer_tc(const MlpDevice& m, const void* image, uint64_t n, float* scores, int* err,
                                cudaStream_t stream)
{
    if (!n) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(mlp_infer_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(kSmTotal));
    if (e != cudaSuccess) return e;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const uint64_t tiles = (n + kTileRows - 1) / kTileRows;
    const uint32_t grid = static_cast<uint32_t>(std::min<uint64_t>(tiles, static_cast<uint64_t>(sms)));
    mlp_infer_kernel<<<grid, kInferThreads, kSmTotal, stream>>>(
        static_cast<const uint8_t*>(image), n, reinterpret_cast<const uint8_t*>(m.w1_bf16),
        reinterpret_cast<const uint8_t*>(m.w2_bf16), m.params, scores, err);
    return cudaGetLastError();
}

cudaError_t mlp_forward_f32(const MlpDevice& m, const MlpWork& w, const float* x, uint64_t n, cudaStream_t st)
{
    const uint32_t H = kMlpHidden, R = static_cast<uint32_t>(n);
    if (!n) return cudaSuccess;
    const dim3 grid(H / kTile, mlp_parts(n).row_tiles);
    // h1 = relu(x . W1^T + b1), h2 = relu(h1 . W2^T + b2)
    gemm_f32_kernel<false, true, Epilogue::kBiasRelu>
        <<<grid, 256, 0, st>>>(x, kMlpIn, m.params + kOffW1, kMlpIn, w.h1, R, H, kMlpIn, kMlpIn, m.params + kOffB1,
                               nullptr, nullptr);
    gemm_f32_kernel<false, true, Epilogue::kBiasRelu>
        <<<grid, 256, 0, st>>>(w.h1, H, m.params + kOffW2, H, w.h2, R, H, H, H, m.params + kOffB2, nullptr, nullptr);
    score_f32_kernel<<<grid_for(n * 32, 256), 256, 0, st>>>(w.h2, m.params, n, w.s);
    return cudaGetLastError();
}

cudaError_t mlp_loss_backward_f32(const MlpDevice& m, const MlpWork& w, const float* x, const float* y,
                                  const float* weight, uint64_t n, cudaStream_t st)
{
    const uint32_t H = kMlpHidden;
    const uint32_t R = static_cast<uint32_t>(n);
    cudaError_t e = cudaMemsetAsync(w.loss, 0, 2 * sizeof(double), st);
    if (e != cudaSuccess) return e;
    loss_kernel<<<grid_for(n, 256), 256, 0, st>>>(w.s, y, weight, n, w.ds, w.loss);
    const MlpParts p = mlp_parts(n);
    float *pw1 = w.parts, *pw2 = pw1 + p.w2, *pb1 = pw1 + p.b1, *pcol = pw1 + p.col;
    backward_columns_kernel<<<p.col_blocks, H, 0, st>>>(w.ds, w.h2, m.params, w.loss, n, w.dh2, pcol);
    // dW2 = dh2^T h1
    gemm_f32_kernel<true, false, Epilogue::kPartial><<<dim3(H / kTile, H / kTile, p.z2), 256, 0, st>>>(
        w.dh2, H, w.h1, H, pw2, H, H, R, p.w2_rows, nullptr, nullptr, nullptr);
    // dh1 = dh2 W2 where h1 > 0; its column sums are db1
    gemm_f32_kernel<false, false, Epilogue::kMask><<<dim3(H / kTile, p.row_tiles), 256, 0, st>>>(
        w.dh2, H, m.params + kOffW2, H, w.dh1, R, H, H, H, nullptr, w.h1, pb1);
    // dW1 = dh1^T x
    gemm_f32_kernel<true, false, Epilogue::kPartial><<<dim3(kMlpIn / kTile, H / kTile, p.z1), 256, 0, st>>>(
        w.dh1, H, x, kMlpIn, pw1, H, kMlpIn, R, p.w1_rows, nullptr, nullptr, nullptr);
    reduce_gradient_kernel<<<(kMlpParams + 255) / 256, 256, 0, st>>>(pw1, p.z1, pw2, p.z2, pb1, p.row_tiles, pcol,
                                                                    p.col_blocks, w.grad);
    return cudaGetLastError();
}

cudaError_t mlp_adam_step(const MlpDevice& m, const float* grad, float* m1, float* m2, float lr, uint32_t step,
                          cudaStream_t st)
{
    const float c1 = 1.f - powf(0.9f, static_cast<float>(step));
    const float c2 = 1.f - powf(0.999f, static_cast<float>(step));
    adam_kernel<<<256, 256, 0, st>>>(m.params, grad, m1, m2, kMlpParams, lr, c1, c2);
    return cudaGetLastError();
}

}  // namespace emp
