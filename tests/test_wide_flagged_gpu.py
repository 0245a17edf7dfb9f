"""Boards whose rows have trials to replay and whose candidate sets take several words: on both sides
of the rule that chooses the default search, it is no slower than the bitfield search, which is the
faster one for some (by 25 %; 10 % is allowed for noise).  Their trees are too big to count; what the two
searches count on such rows is compared with the oracle in test_compact_kernel_cpu.py and
test_compact_flagged_gpu.py."""
from __future__ import annotations

import pytest

from edge_matching_puzzle_b200 import native
from edge_matching_puzzle_b200.puzzle import generate

pytestmark = pytest.mark.gpu

# two words: four and five words of the bitfield search; four words: seven and nine
BOARDS = [(12, 8, 3, 5, 0), (10, 10, 3, 5, 0), (12, 9, 3, 5, 2), (12, 12, 2, 4, 1), (14, 14, 2, 3, 1)]


@pytest.mark.parametrize("board", BOARDS, ids=str)
def test_not_slower_than_the_bitfield_search(board):
    npz = native.NativePuzzle(board[0], board[1], generate(*board).colors)
    rate = {}
    for placement in (0, 3):
        kw = dict(split_depth=6, timeout_ms=300, stack_placement=placement)
        native.bt_count(npz, **kw)
        r = native.bt_count(npz, **kw)
        rate[placement] = (r.nodes - r.expansion_nodes) / r.kernel_ms
    assert rate[0] >= 0.9 * rate[3], rate
