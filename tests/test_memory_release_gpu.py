"""emp_release_memory gives the device memory that is kept between calls back to the driver; live
plans keep theirs and later calls get theirs again."""
from __future__ import annotations

import pytest

from edge_matching_puzzle_b200 import native

pytestmark = pytest.mark.gpu


def test_kept_memory_goes_back():
    torch = pytest.importorskip("torch")
    free = lambda: torch.cuda.mem_get_info()[0]
    puzzle = native.NativePuzzle(8, 8, native.generate(8, 8, 5, 12, 0))
    want = native.bt_count(puzzle).nodes  # modules are loaded, too
    native.release_memory()
    before = free()
    plan = native.BtPlan([puzzle])
    assert native.bt_count(puzzle).nodes == want
    held = before - free()
    assert held >= 64 << 20  # the two plans' queues
    native.release_memory()
    assert free() >= before - held // 2 - (32 << 20)  # the second plan's are back ...
    plan.run()
    assert plan.results()[0].nodes == want  # ... and the first plan's are not
    plan.close()
    native.release_memory()
    assert free() >= before - (32 << 20)
    assert native.bt_count(puzzle).nodes == want
    with pytest.raises(native.EmpError):
        native.release_memory(1000)
