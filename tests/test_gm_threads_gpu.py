"""The threads that share a glutton trial: a pass's candidates are dealt out evenly to the blocks, a block
takes up to 1024 of its share at a time, and m of them are tried by T threads each, the largest power of
two with m * T <= 1024 and at most one thread too many for the board's words of eight pieces.  The
block counts here give every T that a board allows on the first pass, among them m just up to and
just past 1024 / T, and must not change anything: trials, passes and both boards equal those of
one block, and the trajectory the CPU oracle's where that is affordable."""
from __future__ import annotations

import pytest

from edge_matching_puzzle_b200 import native
from edge_matching_puzzle_b200.puzzle import generate
from oracle.oracle import OraclePuzzle

pytestmark = pytest.mark.gpu

# width, height, border and interior colours, pushes, whether the oracle makes them too (seconds)
BOARDS = [(4, 4, 3, 4, 0, True), (6, 7, 3, 6, 4, True), (8, 8, 4, 8, 2, True), (3, 42, 4, 8, 1, True),
          (10, 13, 4, 9, 6, False), (12, 12, 4, 10, 6, False), (16, 16, 5, 17, 4, False)]


def _threads(m, words):
    t = 1
    while t < 32 and 2 * m * t <= 1024 and t < words:
        t *= 2
    return t


def _first_pass(total, words, blocks):
    """(T, whether one more or one candidate fewer has another T) of every step of every block."""
    out = set()
    for b in range(blocks):
        c0, c1 = total * b // blocks, total * (b + 1) // blocks
        while c0 < c1:
            m = min(c1 - c0, 1024)
            t = _threads(m, words)
            out.add((t, "last" if m < 1024 and _threads(m + 1, words) != t else
                     "first" if m > 1 and _threads(m - 1, words) != t else ""))
            c0 += m
    return out


def _block_counts(total, words):
    """Few block counts that between them make every kind of step that any makes."""
    kinds = {n: _first_pass(total, words, n) for n in range(2, 149)}
    left, picked = set().union(*kinds.values()), [148]
    left -= kinds[148]
    while left:
        n = max(kinds, key=lambda k: len(kinds[k] & left))
        picked.append(n)
        left -= kinds[n]
    return picked


def _state(r, n):
    return (r.status, r.max_level, r.level, r.trials, r.pushes, r.pops, r.passes, r.levels,
            list(r.best_board)[:n], list(r.final_board)[:n])


def _board(played, levels, n):
    cells = [0xFFFFFFFF] * n
    for p in list(played)[:levels]:
        if p != 0xFFFFFFFF:
            cells[p & 0xFF] = (((p >> 8) & 0xFF) << 2) | (p >> 16)
    return cells


@pytest.mark.parametrize("board", BOARDS, ids=lambda b: f"{b[0]}x{b[1]}")
def test_block_counts_change_nothing(board):
    w, h, b, i, pushes, oracle = board
    n, words = w * h, (w * h + 7) // 8
    pz = generate(w, h, b, i, 5)
    npz, op = native.NativePuzzle(w, h, pz.colors), OraclePuzzle(w, h, pz.colors)
    total = sum(bin(x).count("1") for row in op.glutton_initial() for x in row)
    counts = _block_counts(total, words)
    seen = {t for c in counts for t, _ in _first_pass(total, words, c)}
    assert len(seen) >= (1 if words < 4 else 4)
    one = native.glutton_max(npz, push_budget=pushes, timeout_ms=60000, blocks=1)
    if oracle:
        want = op.glutton(push_budget=pushes)
        assert (one.status, one.max_level, one.pushes, one.pops, one.levels) == \
            (want.status, want.max_level, want.pushes, want.pops, want.levels_evaluated)
        assert list(one.best_board)[:n] == _board(want.max_played, want.max_level, n)
        assert list(one.final_board)[:n] == _board(want.played, want.level, n)
    for blocks in counts:
        got = native.glutton_max(npz, push_budget=pushes, timeout_ms=60000, blocks=blocks)
        assert _state(got, n) == _state(one, n), blocks
    if n <= 100:
        assert _state(native.glutton_max_noalloc(npz, push_budget=pushes, timeout_ms=60000), n) == _state(one, n)
