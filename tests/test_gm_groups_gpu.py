"""The glutton search at the sizes where its trial groups change (8 lanes up to 64 pieces, 16 up to
128, 32 above) and on boards of odd shapes, against the CPU oracle."""
from __future__ import annotations

import functools

import pytest

from edge_matching_puzzle_b200 import native
from edge_matching_puzzle_b200.puzzle import generate
from oracle.oracle import OraclePuzzle

pytestmark = pytest.mark.gpu

# width, height, border colours, interior colours, push budget
SHAPES = [(2, 2, 1, 1, 0), (2, 3, 1, 1, 0), (7, 9, 3, 6, 6), (8, 8, 4, 8, 6), (5, 13, 3, 7, 4), (2, 33, 3, 3, 8),
          (3, 42, 4, 8, 2), (8, 16, 4, 9, 1), (3, 43, 4, 8, 2)]


@functools.lru_cache(maxsize=None)
def _oracle(shape):
    w, h, b, i, pushes = shape
    return OraclePuzzle(w, h, generate(w, h, b, i, 5).colors).glutton(push_budget=pushes)


@pytest.mark.parametrize("blocks", [1, 3, 0])
@pytest.mark.parametrize("shape", SHAPES)
def test_group_sizes_take_the_oracle_trajectory(shape, blocks):
    w, h, b, i, pushes = shape
    pz = generate(w, h, b, i, 5)
    want = _oracle(shape)
    got = native.glutton_max(native.NativePuzzle(w, h, pz.colors), push_budget=pushes, timeout_ms=60000, blocks=blocks)
    assert (got.status, got.max_level, got.pushes, got.pops, got.levels) == \
        (want.status, want.max_level, want.pushes, want.pops, want.levels_evaluated)
    best = [-1] * pz.nb_pieces
    for level in range(want.max_level):
        pi = want.max_played[level]
        if pi != 0xFFFFFFFF:
            best[pi & 0xFF] = (((pi >> 8) & 0xFF) << 2) | (pi >> 16)
    assert [c if c != 0xFFFFFFFF else -1 for c in list(got.best_board)[: pz.nb_pieces]] == best
