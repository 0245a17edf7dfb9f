"""Performance cases of edge_matching_puzzle_b200: the calls its users make, at the sizes they make them.

  count    whole exhaustive counts of one puzzle (bt_count), smallest to wide boards, row-major and spiral order
  slice    a slice of an 8x8 tree on a plan that is kept (BtPlan.select / run / results, one graph launch per run)
  slices   the same slices of several puzzles through the one-shot call (bt_count_batch), plans built inside the call
  batch    many small puzzles of mixed sides in one graph launch (bt_count_batch with per-puzzle split depths)
  glutton  the greedy max-placement search with a push budget (glutton_max and glutton_max_noalloc)
  score    the candidate network's scores of host feature rows on the tensor cores (Mlp.score)
  grad     the network's loss and whole gradient (Mlp.loss_grad)
  order    a plan's subtrees queued best first by the network, then searched (BtPlan.order, run, subtree_counts)

Counts, boards and trajectories are whole numbers and have no 64-bit value apart from themselves; exact() gives
the network's scores and gradients.
"""
from __future__ import annotations

import numpy as np

from edge_matching_puzzle_b200 import native
from edge_matching_puzzle_b200.puzzle import spiral_order

INPUTS, HIDDEN = native.MLP_INPUTS, native.MLP_HIDDEN

# Interior colours that keep a square board's whole row-major tree countable in a pass, by its longer side,
# and the placements such a tree holds (geometric mean over seeds).
COLOURS = {4: 4, 5: 5, 6: 7, 7: 8, 8: 10, 9: 13, 10: 17}
PLACEMENTS = {4: 2e2, 5: 1.5e3, 6: 2e4, 7: 7e5, 8: 2e7, 9: 1.2e7, 10: 5e7}
# 8x8 puzzles (4 border, 8 interior colours) by seed: placements of their whole trees, 1/64 of which is a slice
TREES_8X8 = {0: 1.76e11, 1: 3.07e10, 2: 1.96e11, 3: 4.81e10, 4: 3.78e9, 6: 5.97e10, 7: 2.04e11, 8: 5.21e10,
             9: 1.41e11, 10: 6.51e10, 11: 4.49e10, 12: 1.9e10, 14: 6.52e10, 15: 1.77e11}
SLICES = 64


def _count(name, w, h, border, interior, order="basic"):
    return {"name": name, "kind": "count", "w": w, "h": h, "border": border, "interior": interior, "order": order}


def listed():
    return [
        # the smallest whole count: 5x5, 3 border and 5 interior colours; a call is all latency
        _count("count 5x5", 5, 5, 3, 5),
        # an ordinary count, and one in the spiral order (levels with three and four placed neighbours)
        _count("count 7x7", 7, 7, 4, 8),
        _count("count 6x6 spiral", 6, 6, 4, 8, "spiral"),
        # a board of 100 pieces: candidate sets several words wide
        _count("count 10x10", 10, 10, 5, 17),
        # the main workload: 1/64 of an 8x8 tree with tables and prefixes resident
        {"name": "slice 8x8", "kind": "slice", "puzzle": 0},
        # the same workload from host puzzles, four trees in one call
        {"name": "slices 8x8 one-shot", "kind": "slices", "puzzles": "1,3,11,14"},
        # throughput over many small instances of uneven size, 4 to 10 interior colours and no fewer than the side
        # (below that a 6x6 tree can hold millions of solutions and takes a deadline instead of a whole count)
        {"name": "batch of 256", "kind": "batch", "count": 256, "most": 6},
        # the greedy search: a small board in the fixed scratch memory on one block, the largest board on the grid
        {"name": "glutton 8x8 noalloc", "kind": "glutton", "side": 8, "border": 4, "interior": 8, "pushes": 150,
         "noalloc": True},
        {"name": "glutton 16x16", "kind": "glutton", "side": 16, "border": 5, "interior": 17, "pushes": 300,
         "noalloc": False},
        # the network on its own: scoring rows, one training batch's gradient, ordering a plan
        {"name": "score 40000", "kind": "score", "rows": 40000},
        {"name": "grad 2048", "kind": "grad", "rows": 2048},
        {"name": "order 7x7", "kind": "order", "side": 7, "border": 4, "interior": 8, "puzzle": 11},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["count", "count", "slice", "slices", "batch", "glutton", "score", "grad", "order"])
    if kind == "count":
        if rng.random() < 0.25:
            side = rng.randint(4, 6)
            c = _count("", side, side, rng.randint(4, 6), 2 * side - 4 + rng.randint(0, 4), "spiral")
        else:
            w = rng.randint(4, 10)
            h = min(10, max(4, w + rng.randint(-2, 2)))
            c = _count("", w, h, rng.randint(4, 6), COLOURS[max(w, h)] + rng.randint(0, 3))
        del c["name"]
        return c
    if kind == "slice":
        return {"kind": kind, "puzzle": rng.choice([s for s, t in TREES_8X8.items() if t <= 1.76e11])}
    if kind == "slices":
        few = [s for s, t in TREES_8X8.items() if t < 6.6e10]
        return {"kind": kind, "puzzles": ",".join(str(s) for s in sorted(rng.sample(few, rng.randint(1, 3))))}
    if kind == "batch":
        return {"kind": kind, "count": _log_int(rng, 12, 256), "most": rng.randint(5, 6)}
    if kind == "glutton":
        side = rng.randint(4, 16)
        return {"kind": kind, "side": side, "border": rng.randint(4, 5), "interior": min(17, side + rng.randint(0, 3)),
                "pushes": _log_int(rng, 20, 300), "noalloc": side <= 10 and rng.random() < 0.5}
    if kind == "score":
        return {"kind": kind, "rows": _log_int(rng, 1, 40000)}
    if kind == "grad":
        return {"kind": kind, "rows": _log_int(rng, 32, 2048)}
    return {"kind": kind, "side": rng.randint(5, 7), "border": rng.randint(4, 5), "interior": rng.randint(8, 9),
            "puzzle": rng.randint(0, 999)}


def _puzzle(w, h, border, interior, seed, order="basic"):
    return native.NativePuzzle(w, h, native.generate(w, h, border, interior, seed),
                               spiral_order(w, h) if order == "spiral" else None)


def _params(rng):
    """Network weights as emp_mlp_create scales them, with small biases as after training."""
    def layer(fan_out, fan_in):
        return (rng.uniform(-1, 1, fan_out * fan_in) / np.sqrt(fan_in)).astype(np.float32)
    return np.concatenate([layer(HIDDEN, INPUTS), layer(HIDDEN, 1) * np.float32(0.05), layer(HIDDEN, HIDDEN),
                           layer(HIDDEN, 1) * np.float32(0.05), layer(1, HIDDEN), layer(1, 1) * np.float32(0.05)])


def _rows(rng, n):
    """Feature rows as candidates give them: one active entry in each of 20 groups of 25 inputs."""
    x = np.zeros((n, INPUTS), dtype=np.float32)
    x[np.arange(n)[:, None], 25 * np.arange(20)[None, :] + rng.integers(0, 25, (n, 20))] = 1.0
    return x


def _network(case, seed):
    """Parameters and inputs of a score or grad case, from the seed alone."""
    rng = np.random.default_rng(seed)
    p = _params(rng)
    x = _rows(rng, case["rows"])
    if case["kind"] == "score":
        return p, x
    return p, x, (rng.random(case["rows"]) < 0.3).astype(np.float32), rng.uniform(
        0.5, 2.0, case["rows"]).astype(np.float32)


class State:
    """What a program has in hand before the call."""

    def __init__(self, case, seed):
        self.case, self.seed, self.kind = case, seed, case["kind"]
        k = self.kind
        if k == "count":
            self.puzzles = [_puzzle(case["w"], case["h"], case["border"], case["interior"], seed, case["order"])]
        elif k == "slice":
            self.puzzles = [_puzzle(8, 8, 4, 8, case["puzzle"])]
            self.plan = native.BtPlan(self.puzzles, split_depth=12, use_graph=1)
            n = self.plan.subtrees()
            self.first = seed % SLICES
            self.count = (n - self.first + SLICES - 1) // SLICES
        elif k == "slices":
            self.puzzles = [_puzzle(8, 8, 4, 8, int(s)) for s in case["puzzles"].split(",")]
        elif k == "batch":
            rng = np.random.default_rng(seed)
            self.puzzles = []
            for _ in range(case["count"]):
                side = int(rng.integers(4, case["most"] + 1))
                self.puzzles.append(_puzzle(side, side, int(rng.integers(3, 6)), int(rng.integers(side, 11)),
                                            int(rng.integers(0, 1 << 62))))
        elif k == "glutton":
            self.puzzles = [_puzzle(case["side"], case["side"], case["border"], case["interior"], seed)]
        elif k in ("score", "grad"):
            p, *self.inputs = _network(case, seed)
            self.model = native.Mlp(seed=1)
            self.model.set_params(p)
        else:
            self.puzzles = [_puzzle(case["side"], case["side"], case["border"], case["interior"], case["puzzle"])]
            self.model = native.Mlp(seed=1)
            self.model.set_params(_params(np.random.default_rng(seed)))
            self.plan = native.BtPlan(self.puzzles, split_depth=12, keep_subtree_counts=1)
            self.count = self.plan.subtrees()


def prepare(case, seed):
    return State(case, seed)


def _of(r):
    """A count's results: the fields that a search defines (times and round counts are not among them)."""
    return [np.array([r.solutions, r.nodes, r.subtrees, r.expansion_nodes], dtype=np.uint64).astype(np.int64),
            np.array([r.status, r.split_depth, r.has_first_solution], dtype=np.int64),
            np.frombuffer(r.first_solution, dtype=np.uint32).astype(np.int64)]


def run(state):
    c, k = state.case, state.kind
    if k == "count":
        return _of(native.bt_count(state.puzzles[0]))
    if k == "slice":
        state.plan.select(state.first, SLICES, state.count)
        state.plan.run()
        return _of(state.plan.results()[0])
    if k == "slices":
        return [_of(r) for r in native.bt_count_batch(state.puzzles, split_depth=12, sample_stride=SLICES,
                                                      sample_first=state.seed % SLICES)]
    if k == "batch":
        res = native.bt_count_batch(state.puzzles, split_subtrees=1024, use_graph=1, table_placement=1)
        return [np.stack(a) for a in zip(*[_of(r) for r in res])]
    if k == "glutton":
        search = native.glutton_max_noalloc if c["noalloc"] else native.glutton_max
        r = search(state.puzzles[0], push_budget=c["pushes"])
        return [np.array([r.status, r.max_level, r.level, r.trials, r.pushes, r.pops, r.passes, r.levels],
                         dtype=np.int64),
                np.frombuffer(r.best_board, dtype=np.uint32).astype(np.int64),
                np.frombuffer(r.final_board, dtype=np.uint32).astype(np.int64)]
    if k == "score":
        return state.model.score(state.inputs[0])
    if k == "grad":
        loss, grads = state.model.loss_grad(*state.inputs)
        return [loss, grads]
    state.plan.order(state.model)
    state.plan.run()
    r = state.plan.results()[0]
    nodes, solutions = state.plan.subtree_counts(state.count)
    return [_of(r), np.array(nodes, dtype=np.int64), np.array(solutions, dtype=np.int64)]


def _search_work(placements, pieces, puzzles=1):
    """A search reads its tables and writes its result; per placement 4 operations a 32-bit word of the placed
    kind's candidate set (select, mask, clear, test) and 8 beside them."""
    words = (4 * pieces + 31) // 32
    return {"bytes": float(puzzles * (pieces * 128 + 1100)), "flops": placements * (4.0 * words + 8.0)}


def work(case):
    k = case["kind"]
    if k == "count":
        side = max(case["w"], case["h"])
        placements = 5e5 if case["order"] == "spiral" else PLACEMENTS[side]
        return _search_work(placements, case["w"] * case["h"])
    if k == "slice":
        return _search_work(TREES_8X8[case["puzzle"]] / SLICES, 64)
    if k == "slices":
        seeds = [int(s) for s in case["puzzles"].split(",")]
        return _search_work(sum(TREES_8X8[s] for s in seeds) / SLICES, 64, len(seeds))
    if k == "batch":  # the few instances of the largest side with the fewest colours hold most of the placements
        return _search_work(case["count"] * (1e5 if case["most"] > 5 else 2e3), case["most"] ** 2, case["count"])
    if k == "glutton":  # a push evaluates the candidates of its level: each position against each piece's turns once
        n = case["side"] ** 2
        return {"bytes": 128.0 * n + 4096, "flops": case["pushes"] * 4.0 * n * 32}
    per_row = 2.0 * (INPUTS * HIDDEN + HIDDEN * HIDDEN + HIDDEN)
    if k == "score":
        return {"bytes": case["rows"] * 4.0 * (INPUTS + 1) + 4.0 * native.MLP_PARAMS, "flops": case["rows"] * per_row}
    if k == "grad":
        return {"bytes": case["rows"] * 4.0 * (INPUTS + 2) + 8.0 * native.MLP_PARAMS,
                "flops": case["rows"] * (3.0 * per_row - 2.0 * INPUTS * HIDDEN)}
    n = case["side"] ** 2
    prefixes = 2e3 * 3 ** (case["side"] - 5)
    return {"bytes": prefixes * (24.0 + 16.0) + 4.0 * native.MLP_PARAMS, "flops": prefixes * 11 * per_row +
            PLACEMENTS[case["side"]] * (4.0 * ((4 * n + 31) // 32) + 8.0)}


def exact(case, seed):
    """Scores and gradients in 64 bits; the searches give whole numbers."""
    if case["kind"] not in ("score", "grad"):
        return None
    p, x, *yw = _network(case, seed)
    p, x = p.astype(np.float64), x.astype(np.float64)
    cut = np.cumsum([HIDDEN * INPUTS, HIDDEN, HIDDEN * HIDDEN, HIDDEN, HIDDEN])
    w1, b1, w2, b2, w3, b3 = np.split(p, cut)
    w1, w2 = w1.reshape(HIDDEN, INPUTS), w2.reshape(HIDDEN, HIDDEN)
    h1 = np.maximum(x @ w1.T + b1, 0)
    h2 = np.maximum(h1 @ w2.T + b2, 0)
    s = h2 @ w3 + b3[0]
    if case["kind"] == "score":
        return s
    y, w = (v.astype(np.float64) for v in yw)
    total = w.sum()
    loss = float((w * (np.logaddexp(0, s) - y * s)).sum() / total)
    ds = w * (1 / (1 + np.exp(-s)) - y) / total
    dh2 = np.outer(ds, w3) * (h2 > 0)
    dh1 = (dh2 @ w2) * (h1 > 0)
    return [loss, np.concatenate([(dh1.T @ x).ravel(), dh1.sum(0), (dh2.T @ h1).ravel(), dh2.sum(0), ds @ h2,
                                  [ds.sum()]])]
