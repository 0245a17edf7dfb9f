"""Boards with so many solutions that lanes of the lowest subtree find them all the time: counts and the
first solution equal the oracle's, and a deadline is kept although every solution is compared with
the recorded one."""
from __future__ import annotations

import functools

import pytest

from edge_matching_puzzle_b200 import native
from edge_matching_puzzle_b200.puzzle import generate
from oracle.oracle import OraclePuzzle

pytestmark = pytest.mark.gpu

# up to one solution in twenty placements
BOARDS = [(5, 5, 1, 2, 381120792), (5, 5, 1, 2, 183144121), (5, 4, 2, 2, 683740563), (6, 5, 2, 2, 140422590)]


@functools.lru_cache(maxsize=None)
def _puzzle(board):
    pz = generate(*board)
    want, _ = OraclePuzzle(pz.width, pz.height, pz.colors).run()
    assert want.solutions > 1000
    return native.NativePuzzle(pz.width, pz.height, pz.colors), want


def _check(r, want, n):
    assert (r.status, r.nodes, r.solutions) == (native.EMP_OK, want.nodes, want.solutions)
    assert list(r.first_solution)[:n] == list(want.first_board)[:n]


@pytest.mark.parametrize("board", BOARDS, ids=str)
@pytest.mark.parametrize("kw", [{}, {"split_budget": 1}, {"split_budget": 1 << 20}, {"table_placement": 1}], ids=str)
def test_first_solution_and_counts(board, kw):
    npz, want = _puzzle(board)
    for depth in (1, 4, 8):
        _check(native.bt_count(npz, split_depth=depth, **kw), want, board[0] * board[1])


def test_a_kept_plan_run_again():
    """The record of an earlier run is not taken for this one's."""
    npz, want = _puzzle(BOARDS[0])
    plan = native.BtPlan([npz], split_depth=6)
    n = plan.subtrees()
    for first in (0, n // 2, 0):
        plan.select(first, 1, n - first)
        plan.run()
        r = plan.results()[0]
        if first == 0:
            assert r.solutions == want.solutions
            assert list(r.first_solution)[:25] == list(want.first_board)[:25]
        else:
            assert r.solutions < want.solutions and r.has_first_solution
            assert list(r.first_solution)[:25] != list(want.first_board)[:25]
    plan.close()


def test_puzzles_of_one_plan():
    handles, want = zip(*[_puzzle(b) for b in BOARDS])
    for b, r, w in zip(BOARDS, native.bt_count_batch(list(handles), split_depth=6), want):
        _check(r, w, b[0] * b[1])


@pytest.mark.parametrize("placement", [1, 3, 4])
@pytest.mark.parametrize("board", BOARDS[:3], ids=str)
def test_bitfield_search(board, placement):
    npz, want = _puzzle(board)
    for budget in (1, 0):
        _check(native.bt_count(npz, split_depth=4, stack_placement=placement, split_budget=budget), want,
               board[0] * board[1])


@pytest.mark.parametrize("placement", [0, 3])
@pytest.mark.parametrize("board", [(7, 7, 1, 2, 0), (10, 10, 1, 2, 1)], ids=str)
def test_deadline(board, placement):
    npz = native.NativePuzzle(board[0], board[1], generate(*board).colors)
    r = native.bt_count(npz, split_depth=6, timeout_ms=200, stack_placement=placement)
    assert r.status == native.EMP_INCOMPLETE
    assert 200 <= r.kernel_ms <= 300  # 4096 steps past the deadline at most; all lanes in a row took 560 to 700 ms
