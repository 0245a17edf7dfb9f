// CPU walk over the compact search tables (csrc/emp_compact.h), step for step what
// dfs_compact_kernel does, with every table and stack access checked: used by
// test_compact_tables.py.  Reads puzzles from standard input, one per line:
//   width height min_nw split_every colours...      (4 * width * height colours)
// and prints per line "nodes solutions", or "none" when the puzzle has no compact tables.
#include "emp_compact.h"

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <vector>

using namespace emp;

namespace {

struct Walk {
    std::vector<uint32_t> b;
    CompactHeader h;
    uint32_t nw = 1;
    uint32_t u32(size_t o) const { return b.at(o); }
    uint64_t u64(size_t o) const { return b.at(o) | static_cast<uint64_t>(b.at(o + 1)) << 32; }
    const uint32_t* desc(uint32_t l) const
    {
        if (l > h.n) std::abort();
        return &b.at(h.desc + 4 * l);
    }
    uint32_t row_at(const uint32_t* d, uint32_t west, uint32_t north) const  // byte offset, checked
    {
        const uint32_t o = d[0] + (west & d[2] & 0xFFFFu) * (row_bytes(nw) / 16) + north * d[1];
        if (o < 4 * h.rows_off || (o - 4 * h.rows_off) % row_bytes(nw) || (o - 4 * h.rows_off) / row_bytes(nw) >= h.rows)
            std::abort();
        return o;
    }
    uint64_t toggle(uint32_t space, uint32_t slot) const
    {
        if (slot >= 64 * nw) std::abort();
        return u64(h.slots + 4 * (space * 64 * nw + slot));
    }
    uint64_t above(uint32_t space, uint32_t slot) const { return u64(h.slots + 4 * (space * 64 * nw + slot) + 2); }
    uint64_t mask(uint32_t row, uint32_t w) const { return u64(row / 4 + 2 * w); }
    uint32_t entry(uint32_t row, uint32_t slot) const
    {
        const uint32_t o = u32(row / 4 + 2 * nw) + 2 * slot;
        if (o < 4 * h.entries || o >= 4 * h.hot) std::abort();
        return (u32(o / 4) >> (8 * (o & 2))) & 0xFFFFu;
    }
};

struct Rec {
    uint32_t len, row, start;
    std::vector<uint64_t> C;
    uint64_t B;
    std::vector<uint32_t> stk;
};

bool any(const std::vector<uint64_t>& r)
{
    for (uint64_t v : r)
        if (v) return true;
    return false;
}

uint32_t first(const std::vector<uint64_t>& r)
{
    for (size_t w = 0; w < r.size(); ++w)
        if (r[w]) return 64 * w + __builtin_ctzll(r[w]);
    std::abort();
}

std::vector<uint64_t> tried(const Walk& k, uint32_t row, std::vector<uint64_t> left)
{
    std::vector<uint64_t> out(k.nw, 0);
    const uint32_t id = k.u32(row / 4 + 2 * k.nw + 1);
    while (any(left)) {
        const uint32_t s = first(left);
        out[s >> 6] |= 1ull << (s & 63);
        left[s >> 6] &= ~(1ull << (s & 63));
        for (uint32_t w = 0; w < k.nw; ++w) left[w] &= ~k.u64(id + 2 * (s * k.nw + w));
    }
    return out;
}

std::vector<uint64_t> candidates(const Walk& k, uint32_t row, uint32_t space, const std::vector<uint64_t>& C, uint64_t B)
{
    std::vector<uint64_t> r(k.nw);
    for (uint32_t w = 0; w < k.nw; ++w) r[w] = k.mask(row, w) & (space ? (w ? 0 : B) : C[w]);
    return k.mask(row, k.nw - 1) >> 63 ? tried(k, row, r) : r;
}

}  // namespace

int main()
{
    unsigned width, height, min_nw, split;
    while (std::scanf("%u %u %u %u", &width, &height, &min_nw, &split) == 4) {
        std::vector<uint8_t> colours(4 * width * height);
        for (uint8_t& c : colours) {
            unsigned v;
            if (std::scanf("%u", &v) != 1) return 1;
            c = static_cast<uint8_t>(v);
        }
        PuzzleModel m;
        std::vector<LevelPlan> plan;
        std::string err;
        if (!build_model(width, height, colours.data(), m, err) || !build_plan(m, order_basic(width, height), plan, err)) {
            std::printf("error %s\n", err.c_str());
            continue;
        }
        Walk k;
        k.b = build_compact(m, plan, min_nw);
        if (k.b.empty()) {
            std::printf("none\n");
            continue;
        }
        std::memcpy(&k.h, k.b.data(), sizeof(k.h));
        k.nw = k.h.nw;
        unsigned long long nodes = 0, sols = 0;
        std::deque<Rec> queue;
        Rec root{0, 0, 0, std::vector<uint64_t>(k.nw), k.u64(k.h.init), std::vector<uint32_t>((k.h.n + 3) & ~3u, 0)};
        for (uint32_t w = 0; w < k.nw; ++w) root.C[w] = k.u64(k.h.init + 2 + 2 * w);
        root.row = k.row_at(k.desc(0), 0, 0);
        queue.push_back(root);
        while (!queue.empty()) {
            Rec s = queue.front();
            queue.pop_front();
            uint32_t L = s.len, row = s.row, space = (k.desc(L)[2] >> 16) & 1u;
            std::vector<uint64_t> R = candidates(k, row, space, s.C, s.B);
            for (uint32_t slot = 0; slot < s.start; ++slot) R[slot >> 6] &= ~(1ull << (slot & 63));
            if (L == 0 && any(R)) {  // position 0 keeps its first transition
                const uint32_t f = first(R);
                R.assign(k.nw, 0);
                R[f >> 6] = 1ull << (f & 63);
            }
            for (unsigned steps = 1;; ++steps) {
                if (!any(R)) {
                    if (L == s.len) break;
                    const uint32_t word = s.stk.at(--L), slot = (word >> 8) & 0xFF;
                    space = (word >> 17) & 1;
                    row = (word >> 14) & 0x3FFF0u;
                    if (space) s.B ^= k.toggle(space, slot);
                    else s.C[slot >> 6] ^= k.toggle(space, slot);
                    if ((word >> 16) & 1) {
                        R = candidates(k, row, space, s.C, s.B);
                        for (uint32_t w = 0; w < k.nw; ++w)
                            R[w] = w < (slot >> 6) ? 0 : w == (slot >> 6) ? R[w] & k.above(space, slot) : R[w];
                        if (!any(R)) std::abort();  // the more bit is exact
                    }
                    if (!any(R)) continue;
                }
                const uint32_t slot = first(R);
                R[slot >> 6] &= R[slot >> 6] - 1;
                const uint32_t e = k.entry(row, slot);
                const uint32_t* d = k.desc(L + 1);
                const uint32_t north = s.stk.at(d[3]) & 0xFFu;
                const uint32_t crow = k.row_at(d, e, north);
                const uint32_t cspace = (d[2] >> 16) & 1u;
                ++nodes;
                std::vector<uint64_t> C = s.C;
                uint64_t B = s.B;
                if (space) B ^= k.toggle(space, slot);
                else C[slot >> 6] ^= k.toggle(space, slot);
                std::vector<uint64_t> c = candidates(k, crow, cspace, C, B);
                if (any(c)) {
                    s.stk.at(L) = (e >> 9) | slot << 8 | static_cast<uint32_t>(any(R)) << 16 | space << 17 | row << 14;
                    s.C = C;
                    s.B = B;
                    ++L;
                    row = crow;
                    space = cspace;
                    R = c;
                } else if (L == k.h.n - 1) {
                    ++sols;
                }
                if (split && steps % split == 0) {  // hand everything back, as split_record does
                    if (any(R)) {
                        Rec r = s;
                        r.len = L;
                        r.row = row;
                        r.start = first(R);
                        queue.push_back(r);
                    }
                    for (uint32_t l = L; l-- > s.len;) {
                        const uint32_t word = s.stk.at(l), q = (word >> 8) & 0xFF, sp = (word >> 17) & 1;
                        if (sp) s.B ^= k.toggle(sp, q);
                        else s.C[q >> 6] ^= k.toggle(sp, q);
                        if (!((word >> 16) & 1)) continue;
                        Rec r = s;
                        r.len = l;
                        r.row = (word >> 14) & 0x3FFF0u;
                        r.start = q + 1;
                        queue.push_back(r);
                    }
                    break;
                }
            }
        }
        std::printf("%llu %llu\n", nodes, sols);
    }
    return 0;
}
