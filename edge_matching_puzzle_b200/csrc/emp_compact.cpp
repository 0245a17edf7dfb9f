// Compact search tables (see emp_compact.h).
#include "emp_compact.h"

#include <algorithm>
#include <array>
#include <cstring>

namespace emp {

namespace {

// one transition of a class: where it is a candidate and what it shows
struct Cand {
    uint16_t t;
    uint8_t west, north, east, south;
};

struct Class {
    uint32_t kind, frame;  // frame sides N,E,S,W as bits 0..3
    bool has_w, has_n;
    std::vector<Cand> cands;             // ascending t
    uint32_t wlo = 31, whi = 0, nlo = 31, nhi = 0;
    uint32_t first_row = 0;
    uint32_t wr() const { return whi - wlo + 1; }
    uint32_t rows() const { return wr() * (nhi - nlo + 1); }
    uint32_t row(uint32_t w, uint32_t n) const { return first_row + (w - wlo) + (n - nlo) * wr(); }
    void see_w(uint32_t c) { wlo = std::min(wlo, c), whi = std::max(whi, c); }
    void see_n(uint32_t c) { nlo = std::min(nlo, c), nhi = std::max(nhi, c); }
};

bool base_bit(const LevelPlan& lp, uint32_t t) { return (lp.base[t >> 5] >> (t & 31)) & 1u; }

}  // namespace

std::vector<uint32_t> build_compact(const PuzzleModel& m, const std::vector<LevelPlan>& plan, uint32_t min_nw)
{
    const uint32_t n = m.n, width = m.width, height = m.height;
    for (uint32_t l = 0; l < n; ++l)
        if (plan[l].position != l) return {};
    // classes of levels
    std::vector<Class> cls;
    std::vector<uint32_t> level_class(n);
    for (uint32_t l = 0; l < n; ++l) {
        const uint32_t x = l % width, y = l / width;
        const uint32_t frame = (y == 0) | (x == width - 1) << 1 | (y == height - 1) << 2 | (x == 0) << 3;
        uint32_t c = 0;
        while (c < cls.size() && cls[c].frame != frame) ++c;
        if (c == cls.size()) {
            // the frame sides fix the kind and which neighbours are placed: west unless x == 0,
            // north unless y == 0
            Class k;
            k.kind = plan[l].kind;
            k.frame = frame;
            k.has_w = x > 0;
            k.has_n = y > 0;
            k.cands.reserve(4 * m.nb_kind(k.kind));
            for (uint32_t t = 0; t < 4 * m.nb_kind(k.kind); ++t) {
                if (!base_bit(plan[l], t)) continue;
                const uint32_t p = m.members[k.kind][t >> 2], o = t & 3u;
                k.cands.push_back({static_cast<uint16_t>(t),
                                   static_cast<uint8_t>(k.has_w ? m.colour(p, 3, o) : 0),
                                   static_cast<uint8_t>(k.has_n ? m.colour(p, 0, o) : 0),
                                   static_cast<uint8_t>(m.colour(p, 1, o)), static_cast<uint8_t>(m.colour(p, 2, o))});
            }
            if (!k.has_w) k.see_w(0);
            if (!k.has_n) k.see_n(0);
            for (const Cand& q : k.cands) {
                k.see_w(q.west);
                k.see_n(q.north);
            }
            cls.push_back(std::move(k));
        }
        level_class[l] = c;
    }
    // colours the placed neighbours can show: rows without candidates are wanted for them too
    for (uint32_t l = 0; l < n; ++l) {
        Class& k = cls[level_class[l]];
        if (k.has_w)
            for (const Cand& q : cls[level_class[l - 1]].cands) k.see_w(q.east);
        if (k.has_n)
            for (const Cand& q : cls[level_class[l - width]].cands) k.see_n(q.south);
    }
    uint32_t rows = 1;  // row 0: no candidate
    for (Class& k : cls) {
        if (k.wlo > k.whi) k.wlo = k.whi = 0;
        if (k.nlo > k.nhi) k.nlo = k.nhi = 0;
        k.first_row = rows;
        rows += k.rows();
    }
    if (rows > 16383) return {};
    // slots: per piece, the largest number of orientations in which one row lists it
    const uint32_t nborder = m.nb_kind(kBorder);
    std::array<std::vector<uint32_t>, 2> need{std::vector<uint32_t>(m.nb_kind(kCenter), 1),
                                              std::vector<uint32_t>(nborder + m.nb_kind(kCorner), 1)};
    auto space_of = [](uint32_t kind) { return kind == kCenter ? 0u : 1u; };
    auto index_of = [&](uint32_t kind, uint32_t ki) { return kind == kCorner ? nborder + ki : ki; };
    for (const Class& k : cls)
        for (size_t i = 0; i < k.cands.size(); ++i) {
            uint32_t same = 1;
            for (size_t j = i; j-- > 0 && (k.cands[j].t >> 2) == (k.cands[i].t >> 2);)
                same += k.cands[j].west == k.cands[i].west && k.cands[j].north == k.cands[i].north;
            uint32_t& w = need[space_of(k.kind)][index_of(k.kind, k.cands[i].t >> 2)];
            w = std::max(w, same);
        }
    // what a trial of candidate a removes of candidate b (both of class k)
    auto removes = [&](const Class& k, const Cand& a, const Cand& b) {
        const uint32_t* im = &m.idmask[k.kind][static_cast<size_t>(a.t) * m.kind_words[k.kind]];
        return !((im[b.t >> 5] >> (b.t & 31)) & 1u);
    };
    // next[s][i]: the next twin of piece i, when every row that lists one of the two lists both and
    // the trials of i in it remove the twin, as do those of any candidate that removes i
    std::array<std::vector<int32_t>, 2> next{std::vector<int32_t>(need[0].size(), -1),
                                             std::vector<int32_t>(need[1].size(), -1)};
    std::array<std::vector<uint8_t>, 2> later{std::vector<uint8_t>(need[0].size(), 0),
                                              std::vector<uint8_t>(need[1].size(), 0)};
    // pieces of one look share the smallest of their four rotated colour words
    std::vector<uint32_t> look(n);
    for (uint32_t p = 0; p < n; ++p) {
        uint32_t c = 0;
        for (uint32_t s = 0; s < 4; ++s) c |= static_cast<uint32_t>(m.colours[p][s]) << (8 * s);
        look[p] = c;
        for (uint32_t o = 8; o < 32; o += 8) look[p] = std::min(look[p], c >> o | c << (32 - o));
    }
    for (uint32_t kind = 0; kind < 3; ++kind) {
        const uint32_t s = space_of(kind);
        for (uint32_t a = 0; a < m.nb_kind(kind); ++a) {
            uint32_t b = a + 1;
            while (b < m.nb_kind(kind) && look[m.members[kind][a]] != look[m.members[kind][b]]) ++b;
            if (b == m.nb_kind(kind) || need[s][index_of(kind, a)] != need[s][index_of(kind, b)]) continue;
            bool ok = true;
            for (const Class& k : cls) {
                if (k.kind != kind || !ok) continue;
                std::vector<const Cand*> pa, pb;
                for (const Cand& q : k.cands) {
                    if ((q.t >> 2) == a) pa.push_back(&q);
                    if ((q.t >> 2) == b) pb.push_back(&q);
                }
                auto row_of = [](const Cand& q) { return q.west << 8 | q.north; };
                for (const Cand* u : pa) {
                    ok = ok && std::any_of(pb.begin(), pb.end(), [&](const Cand* v) { return row_of(*v) == row_of(*u); });
                    for (const Cand& w : k.cands)  // a candidate that removes u removes what u does
                        if (row_of(w) == row_of(*u) && (w.t >> 2) != a && (w.t >> 2) != b && removes(k, w, *u))
                            for (const Cand* v : pb)
                                if (row_of(*v) == row_of(*u) && removes(k, *u, *v)) ok = ok && removes(k, w, *v);
                }
                for (const Cand* v : pb)
                    ok = ok && std::any_of(pa.begin(), pa.end(), [&](const Cand* u) {
                             return row_of(*u) == row_of(*v) && removes(k, *u, *v);
                         });
            }
            if (!ok) continue;
            next[s][index_of(kind, a)] = static_cast<int32_t>(index_of(kind, b));
            later[s][index_of(kind, b)] = 1;
        }
    }
    auto chained = [&](uint32_t s, uint32_t i, uint32_t j) {  // j is a later twin of i
        for (int32_t q = next[s][i]; q >= 0; q = next[s][q])
            if (static_cast<uint32_t>(q) == j) return true;
        return false;
    };
    // a chain's slots lie in one word, so that one mask toggles a piece and its next twin: pieces
    // are numbered in order, and a chain that would straddle words is not used
    std::array<std::vector<uint32_t>, 2> first;
    std::array<uint32_t, 2> nslots{};
    for (uint32_t s = 0; s < 2; ++s)
        for (uint32_t c : need[s]) {
            if ((nslots[s] & 63u) + c > 64) nslots[s] = (nslots[s] + 63) & ~63u;  // a piece stays in one word
            first[s].push_back(nslots[s]);
            nslots[s] += c;
        }
    for (uint32_t s = 0; s < 2; ++s)
        for (size_t i = 0; i < next[s].size(); ++i)
            if (next[s][i] >= 0 && (first[s][i] >> 6) != (first[s][next[s][i]] >> 6)) {
                later[s][next[s][i]] = 0;
                next[s][i] = -1;
            }
    uint32_t nw = std::max(1u, min_nw);
    while (nslots[0] > 64 * nw - 1 && nw < 4) nw *= 2;
    if (nslots[0] > 64 * nw - 1 || nslots[1] > 63) return {};
    const uint32_t cap = 64 * nw;
    // rows
    std::vector<uint64_t> mask(static_cast<size_t>(rows) * nw, 0), toggle(static_cast<size_t>(2) * cap, 0);
    std::vector<int32_t> info(rows, 0);   // entry index of slot 0
    std::vector<uint16_t> entries;
    std::vector<uint32_t> idrow(rows, 0);  // 1 + index into clears of flagged rows
    std::vector<uint64_t> clears;
    uint32_t flagged = 0;
    std::vector<uint8_t> piece(static_cast<size_t>(2) * cap, 0);
    auto piece_bits = [&](uint32_t s, size_t i) { return ((uint64_t(1) << need[s][i]) - 1) << (first[s][i] & 63u); };
    for (uint32_t s = 0; s < 2; ++s)
        for (size_t i = 0; i < need[s].size(); ++i)
            for (uint32_t k = 0; k < need[s][i]; ++k) {
                const uint32_t slot = first[s][i] + k;
                piece[s * cap + slot] = static_cast<uint8_t>(i);
                toggle[s * cap + slot] = piece_bits(s, i) | (next[s][i] >= 0 ? piece_bits(s, next[s][i]) : 0);
            }
    struct In {
        uint32_t row, slot, cand;
    };
    for (const Class& k : cls) {
        const uint32_t s = space_of(k.kind);
        std::vector<In> in;
        in.reserve(k.cands.size());
        for (uint32_t i = 0; i < k.cands.size(); ++i) {
            const Cand& q = k.cands[i];
            uint32_t before = 0;
            for (uint32_t j = i; j-- > 0 && (k.cands[j].t >> 2) == (q.t >> 2);)
                before += k.cands[j].west == q.west && k.cands[j].north == q.north;
            in.push_back({k.row(q.west, q.north), first[s][index_of(k.kind, q.t >> 2)] + before, i});
        }
        std::stable_sort(in.begin(), in.end(), [](const In& a, const In& b) { return a.row < b.row; });
        for (size_t i = 0; i < in.size();) {
            size_t e = i;
            const uint32_t r = in[i].row, lo = in[i].slot;
            while (e < in.size() && in[e].row == r) ++e;
            info[r] = static_cast<int32_t>(entries.size()) - static_cast<int32_t>(lo);
            entries.resize(entries.size() + in[e - 1].slot - lo + 1, 0);
            bool flag = false;
            for (size_t a = i; a < e; ++a) {
                const Cand& q = k.cands[in[a].cand];
                mask[static_cast<size_t>(r) * nw + (in[a].slot >> 6)] |= uint64_t(1) << (in[a].slot & 63u);
                entries[info[r] + in[a].slot] = static_cast<uint16_t>((q.t & 3u) | q.east << 4 | q.south << 9);
                for (size_t b = a + 1; b < e && !flag; ++b) {
                    const Cand& q2 = k.cands[in[b].cand];
                    flag = removes(k, q, q2) &&
                           !chained(s, index_of(k.kind, q.t >> 2), index_of(k.kind, q2.t >> 2));
                }
            }
            if (flag) {
                ++flagged;
                mask[static_cast<size_t>(r) * nw + nw - 1] |= uint64_t(1) << 63;
                const size_t at = clears.size();
                clears.resize(at + static_cast<size_t>(cap) * nw, 0);
                idrow[r] = static_cast<uint32_t>(at) + 1;
                for (size_t a = i; a < e; ++a)
                    for (size_t b = i; b < e; ++b)
                        if (removes(k, k.cands[in[a].cand], k.cands[in[b].cand]))
                            clears[at + static_cast<size_t>(in[a].slot) * nw + (in[b].slot >> 6)] |=
                                uint64_t(1) << (in[b].slot & 63u);
            }
            i = e;
        }
    }
    // layout
    const uint32_t rb = row_bytes(nw);
    CompactHeader h{};
    uint32_t at = kCompactHeader;
    auto place = [&](size_t words, uint32_t align) {
        at = (at + align - 1) / align * align;
        const uint32_t o = at;
        at += static_cast<uint32_t>(words);
        return o;
    };
    h.nw = nw;
    h.n = n;
    h.width = width;
    h.nborder = nborder;
    h.rows = rows;
    h.flagged = flagged;
    h.desc = place(4 * (n + 1), 4);
    h.slots = place(8 * cap, 4);
    h.rows_off = place(static_cast<size_t>(rows) * rb / 4, 4);
    h.entries = place((entries.size() + 1) / 2, 1);
    h.hot = place(0, 4);
    h.init = place(2 * (1 + nw), 2);
    h.piece = place(piece.size() / 4, 1);
    h.first = place(2 * 256 / 4, 1);
    const uint32_t clears_at = place(2 * clears.size(), 2);
    h.words = place(0, 4);
    if (h.hot > 64 * 1024) return {};  // 256 KB
    std::vector<uint32_t> b(h.words, 0);
    std::memcpy(b.data(), &h, sizeof(h));
    for (uint32_t l = 0; l <= n; ++l) {
        uint32_t* d = &b[h.desc + 4 * l];
        d[0] = 4 * h.rows_off;
        if (l == n) break;
        const Class& k = cls[level_class[l]];
        const int32_t base = static_cast<int32_t>(k.first_row) - static_cast<int32_t>(k.has_w ? k.wlo : 0) -
                             static_cast<int32_t>(k.has_n ? k.nlo * k.wr() : 0);
        d[0] += static_cast<uint32_t>(base * static_cast<int32_t>(rb));
        d[1] = k.has_n ? k.wr() * rb : 0;
        d[2] = (k.has_w ? 0x1F0u : 0u) | space_of(k.kind) << 16;
        d[3] = k.has_n ? l - width : 0;
    }
    for (uint32_t i = 0; i < 2 * cap; ++i) {
        const uint32_t bit = i & 63u;
        const uint64_t above = bit == 63 ? 0 : ~uint64_t(0) << (bit + 1);
        std::memcpy(&b[h.slots + 4 * i], &toggle[i], 8);
        std::memcpy(&b[h.slots + 4 * i + 2], &above, 8);
    }
    for (uint32_t r = 0; r < rows; ++r) {
        uint32_t* w = &b[h.rows_off + r * rb / 4];
        std::memcpy(w, &mask[static_cast<size_t>(r) * nw], 8 * nw);
        w[2 * nw] = 4 * h.entries + static_cast<uint32_t>(2 * info[r]);
        w[2 * nw + 1] = idrow[r] ? clears_at + 2 * (idrow[r] - 1) : 0;
    }
    if (!entries.empty()) std::memcpy(&b[h.entries], entries.data(), 2 * entries.size());
    for (uint32_t s = 0; s < 2; ++s) {
        uint64_t* init = reinterpret_cast<uint64_t*>(&b[h.init]);
        for (size_t i = 0; i < need[s].size(); ++i) {
            const uint32_t slot = first[s][i];
            if (!later[s][i]) init[s == 1 ? 0 : 1 + (slot >> 6)] |= piece_bits(s, i);
            reinterpret_cast<uint8_t*>(&b[h.first])[256 * s + i] = static_cast<uint8_t>(slot);
        }
    }
    std::memcpy(&b[h.piece], piece.data(), piece.size());
    if (!clears.empty()) std::memcpy(&b[clears_at], clears.data(), 8 * clears.size());
    return b;
}

}  // namespace emp
