"""The prefix expansion that takes its first levels in one launch: the prefixes of a plan, their order
and their counts equal the oracle's at every split depth, on both sides of the 4096 prefixes
at which it goes on level by level, and for trees that end above the split depth."""
from __future__ import annotations

import pytest

from edge_matching_puzzle_b200 import native
from edge_matching_puzzle_b200.puzzle import generate
from oracle.oracle import OraclePuzzle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depth", [1, 2, 7, 8, 9, 10, 11, 12])
@pytest.mark.parametrize("shape", [(7, 7, 4, 8, 11), (6, 6, 3, 4, 5), (4, 4, 3, 6, 1)])
def test_prefixes_equal_the_oracle(shape, depth):
    w, h, b, i, seed = shape
    pz = generate(w, h, b, i, seed)
    n, nodes, _, want = OraclePuzzle(w, h, pz.colors).expand(depth, max_prefixes=1 << 40)
    plan = native.BtPlan([native.NativePuzzle(w, h, pz.colors)], split_depth=depth)
    assert plan.subtrees() == n
    for k in sorted({0, 1, 1023, 1024, 4095, 4096, n // 2, n - 1}):
        if 0 <= k < n:
            assert plan.subtree_prefix(k, depth) == [int(v) for v in want[k * depth:(k + 1) * depth]], k
    plan.run()
    assert plan.results()[0].expansion_nodes == nodes
    plan.close()
