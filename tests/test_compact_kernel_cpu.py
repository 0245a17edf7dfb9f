"""The compact search's kernel itself (csrc/emp_btc.cu) on the CPU: compact_kernel_host.cpp runs its
source with 128 lanes of one block, warp collectives included, so that the paths hardly any count
on a GPU takes are counted against the oracle: full item queues, stops and superseded subtrees on
rows whose trials are replayed (half-symmetric pieces, few colours), lanes of a warp sharing work."""
from __future__ import annotations

import os
import subprocess

import pytest

from edge_matching_puzzle_b200.puzzle import Puzzle, generate
from oracle.oracle import OraclePuzzle

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "edge_matching_puzzle_b200", "csrc")


@pytest.fixture(scope="module")
def kernel(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("kernel") / "compact_kernel_host")
    subprocess.run(["g++", "-O1", "-std=c++17", "-w", "-U_FORTIFY_SOURCE", "-I/usr/local/cuda/include",
                    "-I" + os.path.join(ROOT, "include"), "-I" + CSRC, "-o", exe,
                    os.path.join(ROOT, "tests", "compact_kernel_host.cpp"), os.path.join(CSRC, "emp_compact.cpp"),
                    os.path.join(CSRC, "emp_model.cpp")], check=True)

    def run(puzzles, depth, smem=0, min_nw=1, budget=256, capacity=1 << 16, deadline=0, at_first=0, at_any=0,
            before=()):
        """Per puzzle (placements, solutions, incomplete) of its subtrees, then the run's clock,
        rounds and rounds with a full queue; and the oracle's (placements, solutions).  before:
        prefixes of the first puzzle that are queued ahead of its subtrees."""
        records = [f"0 {len(p)} " + " ".join(str(t) for t in p) for p in before]
        want = []
        text = [f"{int(smem)} {min_nw} {budget} {capacity} {deadline} {at_first} {at_any}", str(len(puzzles))]
        for i, p in enumerate(puzzles):
            text.append(f"{p.width} {p.height} " + " ".join(str(c) for q in p.colors for c in q))
            op = OraclePuzzle(p.width, p.height, p.colors)
            n, _, _, prefixes = op.expand(depth, max_prefixes=1 << 20)
            records += [f"{i} {depth} " + " ".join(str(t) for t in prefixes[j * depth:(j + 1) * depth])
                        for j in range(n)]
            if not (deadline or at_any or before):  # else not searched out
                want.append(op.subtrees_parallel(prefixes, depth, 0, n, 4))
        text.append(str(len(records)))
        out = subprocess.run([exe], input="\n".join(text + records) + "\n", capture_output=True, text=True,
                             check=True, timeout=120).stdout.splitlines()
        assert out and out[-1].startswith("end"), out
        _, clock, _, rounds, _, full = out[-1].split()
        return [tuple(int(v) for v in l.split()) for l in out[:-1]], (int(clock), int(rounds), int(full)), want
    return run


# boards with half-symmetric pieces: most of their rows have trials to replay
FLAGGED = [(4, 5, 3, 2, 646579118), (5, 5, 2, 2, 338252669), (5, 4, 2, 2, 683740563), (5, 5, 1, 2, 381120792)]


@pytest.mark.parametrize("kw", [{}, {"smem": 1}, {"budget": 1}, {"budget": 1 << 20}, {"min_nw": 2, "budget": 48},
                                {"min_nw": 4, "budget": 48}], ids=str)
def test_counts_equal_oracle(kernel, kw):
    for board in FLAGGED + [(6, 5, 3, 4, 3)]:
        got, _, want = kernel([generate(*board)], 4, **kw)
        assert got == [want[0] + (0,)], board


@pytest.mark.parametrize("board", FLAGGED, ids=str)
@pytest.mark.parametrize("budget,capacity", [(1, 20), (48, 100), (48, 40)])
def test_full_queue_of_flagged_rows(kernel, board, budget, capacity):
    """Lanes that handed work back take it again from their neighbours that could not."""
    for depth in (2, 4):
        for min_nw in (1, 2):
            got, (_, _, full), want = kernel([generate(*board)], depth, budget=budget, capacity=capacity, min_nw=min_nw)
            assert full
            assert got == [want[0] + (0,)], (depth, min_nw)


def _without_solution(w, h, b, i, seed):
    """A generated board with one side of its first centre piece in another side's colour."""
    pz = generate(w, h, b, i, seed)
    cols = [list(q) for q in pz.colors]
    q = next(q for q in cols if 0 not in q)
    q[0] = q[1] if q[1] != q[0] else q[2]
    return Puzzle(w, h, cols)


@pytest.mark.parametrize("first,second,depth,budget", [
    ((6, 5, 2, 2, 140422590), (5, 6, 3, 4, 318208215), 4, 256),
    ((5, 5, 2, 2, 389397901), (6, 5, 3, 4, 435610963), 3, 1 << 20),
    ((5, 5, 1, 2, 472049899), (5, 6, 1, 2, 400191967), 4, 1 << 20)], ids=str)
def test_superseded_lanes_leave_other_puzzles_counts_whole(kernel, first, second, depth, budget):
    """Stop at first: the second puzzle has no solution, so its count is that of its whole tree."""
    got, _, want = kernel([generate(*first), _without_solution(*second)], depth, budget=budget, at_first=1)
    assert want[1][1] == 0
    assert got[1] == want[1] + (0,)
    assert got[0][1]


# ticks in which each of the four warps makes the steps between a lane's looks at the flags (4096, and a
# fetch before and after): a step has at most four collectives
LOOK = 4 * 4 * (4096 + 2 * 48)


@pytest.mark.parametrize("kw", [{"budget": 1 << 20}, {"budget": 256, "capacity": 60}], ids=str)
@pytest.mark.parametrize("board,depth", [((6, 6, 4, 2, 476079230), 5), ((6, 7, 2, 5, 916256161), 3)], ids=str)
def test_deadline_ends_a_run_that_shares_work(kernel, board, depth, kw):
    """Work that a lane at the deadline takes from a neighbour would go on for as long again."""
    deadline = 40000
    got, (clock, _, _), _ = kernel([generate(*board)], depth, deadline=deadline, **kw)
    assert got[0][2] == 1  # incomplete
    assert deadline < clock <= deadline + LOOK


@pytest.mark.parametrize("stop", ["at_first", "at_any"])
@pytest.mark.parametrize("board,depth", [((6, 6, 4, 2, 476079230), 5), ((6, 7, 2, 5, 916256161), 3)], ids=str)
def test_first_solution_ends_a_run_that_shares_work(kernel, board, depth, stop):
    """A first record that holds little but a solution, then subtrees that are not searched out."""
    pz = generate(*board)
    op = OraclePuzzle(pz.width, pz.height, pz.colors)
    r, _ = op.run(node_limit=100000000)
    assert r.solutions
    kinds = {op.piece_of(k, i): i for k in range(3) for i in range(op.nb_kind(k))}
    path = [(kinds[v >> 2] << 2) | (v & 3) for v in list(r.first_board)[: pz.nb_pieces]]
    got, (clock, _, _), _ = kernel([pz], depth, budget=1 << 20, before=[path[:-4]], **{stop: 1})
    assert got[0][1] >= 1
    assert clock <= LOOK
