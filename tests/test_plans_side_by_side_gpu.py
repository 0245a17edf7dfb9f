"""Plans of the bitfield search that exist side by side, a later one with less shared memory than an
earlier one of the same kernel: one call with several puzzles, and plans kept by the caller, give the
oracle's counts."""
from __future__ import annotations

import functools

import pytest

from edge_matching_puzzle_b200 import native
from edge_matching_puzzle_b200.puzzle import generate, spiral_order
from oracle.oracle import OraclePuzzle

pytestmark = pytest.mark.gpu

# width, height, border and interior colours, seed, spiral: descending shared memory
SPIRALS = [(7, 7, 5, 12, 0, True), (6, 7, 5, 12, 1, True), (6, 6, 5, 10, 2, True)]
ROWS = [(7, 7, 5, 13, 3, False), (7, 7, 4, 9, 4, False), (6, 7, 4, 9, 5, False), (6, 6, 4, 8, 6, False)]


@functools.lru_cache(maxsize=None)
def _puzzle(s):
    w, h, b, i, seed, spiral = s
    pz = generate(w, h, b, i, seed)
    order = spiral_order(w, h) if spiral else None
    want = OraclePuzzle(w, h, pz.colors).run(order=order)[0]
    return native.NativePuzzle(w, h, pz.colors, order=order), (native.EMP_OK, want.nodes, want.solutions)


CASES = [(SPIRALS, {}), (SPIRALS, {"threads_per_block": 256}), (SPIRALS, {"stack_placement": 4}),
         *[(ROWS, {"stack_placement": p}) for p in (1, 2, 3, 4)],
         (ROWS, {"stack_placement": 1, "threads_per_block": 256, "table_placement": 2})]


@pytest.mark.parametrize("shapes,kw", CASES, ids=lambda v: str(v) if isinstance(v, dict) else f"{len(v)}")
def test_one_call(shapes, kw):
    handles, want = zip(*[_puzzle(s) for s in shapes])
    for k in (2, len(shapes)):
        got = native.bt_count_batch(list(handles[:k]), split_depth=6, **kw)
        assert [(r.status, r.nodes, r.solutions) for r in got] == list(want[:k])


@pytest.mark.parametrize("shapes,kw", CASES, ids=lambda v: str(v) if isinstance(v, dict) else f"{len(v)}")
@pytest.mark.parametrize("use_graph", [0, 1])
def test_kept_plans(shapes, kw, use_graph):
    plans = [(native.BtPlan([_puzzle(s)[0]], split_depth=6, use_graph=use_graph, **kw), _puzzle(s)[1]) for s in shapes]
    for plan, want in plans:
        plan.run()
        r = plan.results()[0]
        assert (r.status, r.nodes, r.solutions) == want
    for plan, _ in plans:
        plan.close()
