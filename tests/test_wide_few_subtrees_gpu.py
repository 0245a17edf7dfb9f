"""Few subtrees of wide boards of few colours: their threads hand back an item for each of some 40
open levels, and the next round's queue has to hold them all.  A round that found it full went on
with the threads that kept their work, at a tenth of the bitfield search's rate; now the default
search counts at least half as much in the same time (more, by measurement; half leaves room for noise)."""
from __future__ import annotations

import pytest

from edge_matching_puzzle_b200 import native
from edge_matching_puzzle_b200.puzzle import generate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("board", [(12, 8, 3, 5, 0), (10, 10, 3, 5, 0), (12, 12, 4, 6, 0), (14, 14, 5, 16, 1)], ids=str)
def test_rate_is_not_lost_to_a_full_queue(board):
    npz = native.NativePuzzle(board[0], board[1], generate(*board).colors)
    rate = {}
    for placement in (0, 3):
        kw = dict(split_depth=6, timeout_ms=300, stack_placement=placement)
        native.bt_count(npz, **kw)
        r = native.bt_count(npz, **kw)
        assert r.status == native.EMP_INCOMPLETE
        rate[placement] = (r.nodes - r.expansion_nodes) / r.kernel_ms
    assert rate[0] >= 0.5 * rate[3], rate
