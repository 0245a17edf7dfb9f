"""The compact search's kernels (csrc/emp_btc.cu) against the oracle, count for count: candidate
sets of one, two and four words, tables staged in shared memory and read from global memory, every
block size, stacks in shared memory and (12x12, 14x14: too few blocks fit) in global memory, work
handed back after every look at the queue and hardly ever.  Boards of more than 64 centre pieces are
in the second half of the list; four words (14x14) are counted over a sample of subtrees."""
from __future__ import annotations

import functools

import pytest

from edge_matching_puzzle_b200 import native
from edge_matching_puzzle_b200.puzzle import generate, spiral_order
from oracle.oracle import OraclePuzzle

pytestmark = pytest.mark.gpu

# (width, height, border colours, interior colours, seed): whole trees of up to 5e7 placements
BOARDS = [(2, 2, 2, 2, 0), (3, 2, 2, 2, 1), (8, 8, 5, 12, 0), (9, 9, 8, 20, 1), (10, 10, 8, 21, 1), (12, 9, 9, 21, 0),
          (12, 12, 9, 21, 0)]


@functools.lru_cache(maxsize=None)
def _board(b):
    pz = generate(*b)
    want, _ = OraclePuzzle(pz.width, pz.height, pz.colors).run()
    return native.NativePuzzle(pz.width, pz.height, pz.colors), pz.nb_pieces, want


KW = [{}, {"threads_per_block": 128}, {"threads_per_block": 256}, {"threads_per_block": 512}, {"table_placement": 1},
      {"table_placement": 1, "split_budget": 1}, {"split_budget": 1}, {"split_budget": 1 << 20}]


@pytest.mark.parametrize("board", BOARDS, ids=lambda b: f"{b[0]}x{b[1]}")
@pytest.mark.parametrize("kw", KW, ids=str)
def test_counts_equal_oracle(board, kw):
    npz, n, want = _board(board)
    for depth in {1, min(5, n - 1), 0}:
        r = native.bt_count(npz, split_depth=depth, **kw)
        assert r.status == native.EMP_OK
        assert (r.nodes, r.solutions) == (want.nodes, want.solutions), depth
        assert bool(r.has_first_solution) == bool(want.solutions)
        if want.solutions:
            assert list(r.first_solution)[:n] == list(want.first_board)[:n], depth


@functools.lru_cache(maxsize=None)
def _wide(depth, sample):
    pz = generate(14, 14, 8, 22, 0)
    npz = native.NativePuzzle(14, 14, pz.colors)
    op = OraclePuzzle(14, 14, pz.colors)
    plan = native.BtPlan([npz], split_depth=depth)
    total = plan.subtrees()
    assert total == op.expand(depth, max_prefixes=1 << 40)[0]
    stride = total // sample
    plan.select(3, stride, sample)
    return npz, stride, [op.subtree(plan.subtree_prefix(i, depth))[:2] for i in range(sample)]


@pytest.mark.parametrize("kw", KW, ids=str)
def test_four_words_sampled_subtrees(kw):
    depth, sample = 8, 24
    npz, stride, want = _wide(depth, sample)
    plan = native.BtPlan([npz], split_depth=depth, keep_subtree_counts=1, **kw)
    plan.select(3, stride, sample)
    plan.run()
    res = plan.results()[0]
    nodes, sols = plan.subtree_counts(sample)
    assert list(zip(nodes, sols)) == want
    assert (res.nodes, res.solutions) == (sum(nodes), sum(sols))


@pytest.mark.parametrize("count", [2, 4, 5, 11])
@pytest.mark.parametrize("kw", [{}, {"keep_subtree_counts": 1, "split_budget": 1}, {"stack_placement": 1},
                                {"timeout_ms": 60000}], ids=str)
def test_puzzles_side_by_side_equal_oracle(count, kw):
    """A call with a few bigger puzzles runs their searches side by side, in groups: wide boards, a
    spiral order and trees of very different sizes in one call."""
    shapes = [(8, 8, 5, 12, 0), (6, 6, 4, 8, 1), (9, 9, 8, 20, 1), (12, 9, 9, 21, 0), (6, 7, 4, 9, 2), (10, 10, 8, 21, 1),
              (6, 6, 4, 7, 4), (8, 8, 5, 12, 1), (7, 7, 4, 9, 3), (6, 6, 4, 8, 5), (9, 9, 8, 20, 2)]
    pzs = [generate(*b) for b in shapes[:count]]
    orders = [spiral_order(p.width, p.height) if i % 5 == 1 else None for i, p in enumerate(pzs)]
    want = [OraclePuzzle(p.width, p.height, p.colors).run(order=o)[0] for p, o in zip(pzs, orders)]
    handles = [native.NativePuzzle(p.width, p.height, p.colors, order=o) for p, o in zip(pzs, orders)]
    got = native.bt_count_batch(handles, split_depth=8, **kw)
    assert [(r.status, r.nodes, r.solutions) for r in got] == [(native.EMP_OK, w.nodes, w.solutions) for w in want]
    for p, r, w in zip(pzs, got, want):
        if w.solutions:
            assert list(r.first_solution)[: p.nb_pieces] == list(w.first_board)[: p.nb_pieces]
