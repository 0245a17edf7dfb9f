// Compact search tables of the exhaustive backtracker for row-major orders
// (kernel: emp_btc.cu).
//
// In a row-major order the placed neighbours of a position are the one to the west (the
// previous level) and the one to the north (`width` levels before), so a level's
// candidates depend on two colours and a "row" (class of the level, west colour, north
// colour) lists each matching piece in nearly always one orientation: the colours of two
// adjacent sides fix it.  A row's candidates are therefore kept as a set of pieces
// ("slots"), not of piece x orientation: 64 slots per 64-bit word instead of 16 pieces.  A
// piece that matches some row in k orientations (repeated colours) has k consecutive slots,
// used in ascending orientation; placing it takes all of them from the availability.
// Slots ascend with the transition number t = kind_index*4 + orientation inside every row,
// so the lowest set bit is the reference's next candidate (emp_position_strategy.h:205-208).
//
// Twins (pieces that look the same) need no care at a step: only the first unplaced one of a
// chain of twins is available, since the reference tries it first and its trial removes the
// others (emp_position_strategy.h:197-200).  Placing a piece toggles its own bits and those of
// the next twin in the availability, and so does giving it back.  Rows in which one trial
// removes other candidates than twins (a half-symmetric piece's mask, emp_piece.h:208-220)
// are flagged, and their trials are replayed one by one.
//
// Two slot spaces: 0 centre pieces (NW 64-bit words), 1 border and corner pieces together (one
// word).  The flag is bit 63 of a row's last word, so a space of w words holds 64*w - 1 slots.
//
// The blob, 32-bit words; the header's table offsets count words, the offsets inside the tables
// bytes, all from the blob's start:
//   header (kCompactHeader words, CompactHeader below)
//   desc[n + 1]        per level, 4 words: x byte offset of the row of colours 0, 0; y bytes a
//                      north colour steps; z 0x1F0 when a west colour counts | space << 16;
//                      w level of the north neighbour (0: none).  The level's row is at
//                      x + (west entry & z) * (row bytes / 16) + north colour * y.
//                      Level n is the end: the empty row.
//   slots[2][64*NW]    per space and slot, 4 words: what placing it toggles in the word that
//                      holds it (its piece's slots and the next twin's), and the bits above
//                      the slot in that word
//   rows               row_bytes(NW) each, row 0 empty: NW candidate words (with the flag), byte
//                      offset of slot 0 in the entries, word offset of the row's clears
//   entries            16 bits per slot of a row: orientation | east colour << 4 | south colour << 9
//                      (only the slots of the row itself are there)
//   -- the words up to here (hot) may be staged in shared memory --
//   init[1 + NW]       availability of the border space and of the centre space (64 bits)
//                      without the later twins
//   piece[2][64*NW]    bytes: the slot's kind index (border space: corners after the borders)
//   first[2][256]      bytes: first slot of kind index i (space 0: centre, 1: border then corner)
//   clears             flagged rows: [64*NW][NW], per slot the slots its trial removes
#pragma once

#include "emp_model.h"

#include <cstdint>
#include <vector>

namespace emp {

constexpr uint32_t kCompactHeader = 16;

struct CompactHeader {
    uint32_t nw;         // 64-bit words of the centre space
    uint32_t n, width;
    uint32_t desc, slots, rows_off, entries;  // word offsets
    uint32_t hot;        // words of the part a kernel may stage in shared memory (multiple of 4)
    uint32_t init, piece, first;
    uint32_t nborder;    // border pieces: kind index of the first corner in space 1
    uint32_t words;      // blob size (multiple of 4)
    uint32_t rows;
    uint32_t flagged;    // rows whose trials are replayed
    uint32_t pad;
};

constexpr uint32_t row_bytes(uint32_t nw) { return nw == 1 ? 16 : (nw == 2 ? 32 : 48); }

static_assert(sizeof(CompactHeader) == 4 * kCompactHeader, "header words");

// Builds the tables with a centre space of at least min_nw words.  Returns an empty vector
// when the puzzle has no compact form: an order that is not row-major, a border space above
// 63 slots, a centre space above 255, or tables past 256 KB (14 bits of 16-byte steps in a stack
// word).
std::vector<uint32_t> build_compact(const PuzzleModel& m, const std::vector<LevelPlan>& plan, uint32_t min_nw = 1);

}  // namespace emp
