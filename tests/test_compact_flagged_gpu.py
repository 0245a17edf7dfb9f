"""The compact search on boards of few colours, most of whose rows have trials to replay
(half-symmetric pieces), against the oracle: every way work is shared and handed back, and a plan
of several puzzles that stops at first solutions, whose unsolvable puzzle is counted whole."""
from __future__ import annotations

import functools

import pytest

from edge_matching_puzzle_b200 import native
from edge_matching_puzzle_b200.puzzle import Puzzle, generate
from oracle.oracle import OraclePuzzle

pytestmark = pytest.mark.gpu

BOARDS = [(4, 5, 3, 2, 646579118), (5, 5, 2, 2, 338252669), (5, 4, 2, 2, 683740563), (6, 5, 3, 4, 3)]


@functools.lru_cache(maxsize=None)
def _counts(board):
    pz = generate(*board)
    want, _ = OraclePuzzle(pz.width, pz.height, pz.colors).run()
    return native.NativePuzzle(pz.width, pz.height, pz.colors), (want.nodes, want.solutions)


@pytest.mark.parametrize("board", BOARDS, ids=str)
@pytest.mark.parametrize("kw", [{}, {"split_budget": 1}, {"split_budget": 1 << 20}, {"blocks_per_sm": 1},
                                {"table_placement": 1, "split_budget": 1}, {"threads_per_block": 256}], ids=str)
def test_counts_equal_oracle(board, kw):
    npz, want = _counts(board)
    for depth in (1, 3, 8):
        r = native.bt_count(npz, split_depth=depth, **kw)
        assert (r.status, r.nodes, r.solutions) == (native.EMP_OK, *want), depth


@pytest.mark.parametrize("kw", [{}, {"split_budget": 1 << 20}, {"blocks_per_sm": 1, "split_budget": 48}], ids=str)
def test_stop_at_first_counts_unsolvable_puzzles_whole(kw):
    pzs = [generate(6, 5, 2, 2, 140422590), generate(5, 6, 3, 4, 318208215), generate(6, 5, 3, 4, 435610963)]
    for k in (1, 2):  # one side of the first centre piece in another side's colour
        cols = [list(q) for q in pzs[k].colors]
        q = next(q for q in cols if 0 not in q)
        q[0] = q[1] if q[1] != q[0] else q[2]
        pzs[k] = Puzzle(pzs[k].width, pzs[k].height, cols)
    want = [OraclePuzzle(p.width, p.height, p.colors).run()[0] for p in pzs]
    assert want[1].solutions == want[2].solutions == 0
    handles = [native.NativePuzzle(p.width, p.height, p.colors) for p in pzs]
    got = native.bt_count_batch(handles, split_depth=4, stop_at_first=1, **kw)
    assert [(r.status, r.nodes, r.solutions) for r in got[1:]] == [(native.EMP_OK, w.nodes, 0) for w in want[1:]]
    assert list(got[0].first_solution)[:30] == list(want[0].first_board)[:30]


@pytest.mark.parametrize("depth", [3, 12])
def test_deadline_with_work_shared_in_warps(depth):
    """Few subtrees, so that idle lanes take work all the time, and a split budget that hands none
    back.  A lane looks at the clock every 4096 steps (2.3 ms on a full chip): the run ends within
    20 ms of its deadline."""
    pz = generate(8, 8, 4, 8, 0)  # 1.8e11 placements, over a second
    r = native.bt_count(native.NativePuzzle(8, 8, pz.colors), split_depth=depth, timeout_ms=100, split_budget=1 << 20)
    assert r.status == native.EMP_INCOMPLETE
    assert 100 <= r.kernel_ms <= 120
