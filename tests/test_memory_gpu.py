"""Device memory of one-shot calls: freed memory stays in the library's pool up to its limit, calls
from several threads at once get the counts of calls one after the other, and plans of
different sizes can be run in any order."""
from __future__ import annotations

import threading

import pytest

from edge_matching_puzzle_b200 import native
from edge_matching_puzzle_b200.puzzle import generate, spiral_order

pytestmark = pytest.mark.gpu

SHAPES = [(5, 5, 3, 5, 0, None), (6, 6, 4, 8, 1, "spiral"), (7, 7, 4, 8, 2, None), (8, 8, 5, 10, 3, None)]


def _handle(w, h, b, i, seed, order):
    return native.NativePuzzle(w, h, generate(w, h, b, i, seed).colors, spiral_order(w, h) if order else None)


def test_freed_memory_kept_is_bounded():
    torch = pytest.importorskip("torch")
    handles = [_handle(*s) for s in SHAPES]
    native.bt_count(handles[0])
    before = torch.cuda.mem_get_info()[0]
    for _ in range(3):
        for h in handles:
            native.bt_count(h)
    # the pool keeps at most 2 GiB; a quarter as much again for what the driver keeps beside it
    assert before - torch.cuda.mem_get_info()[0] <= 2560 << 20


def test_counts_from_several_threads():
    handles = [_handle(*s) for s in SHAPES]
    want = [(r.nodes, r.solutions) for r in (native.bt_count(h) for h in handles)]
    got = [[None] * len(SHAPES) for _ in range(4)]

    def work(k):
        mine = [_handle(*s) for s in SHAPES]
        for j in range(len(SHAPES)):
            i = (j + k) % len(SHAPES)
            r = native.bt_count(mine[i])
            got[k][i] = (r.nodes, r.solutions)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert got == [want] * 4


@pytest.mark.parametrize("use_graph", [0, 1])
def test_plans_of_several_sizes_run_in_any_order(use_graph):
    handles = [_handle(*s) for s in SHAPES]
    plans = [native.BtPlan([h], use_graph=use_graph) for h in handles]
    want = [native.bt_count(h).nodes for h in handles]
    for order in ([3, 0, 2, 1], [0, 1, 2, 3]):
        for i in order:
            plans[i].run()
            assert plans[i].results()[0].nodes == want[i]
    for p in plans:
        p.close()
