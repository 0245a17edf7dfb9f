"""The compact search tables (csrc/emp_compact.cpp) on the CPU: compact_search.cpp walks them as
the GPU search does, with every access checked, and its counts equal the reference build's and
the oracle's: identical pieces and their asymmetric masks, pieces listed in several orientations
of one row, boards from 2x2 up, one to four words of centre slots, work handed back."""
from __future__ import annotations

import json
import os
import random
import subprocess

import pytest

from edge_matching_puzzle_b200.puzzle import Puzzle, generate
from oracle.oracle import OraclePuzzle

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "edge_matching_puzzle_b200", "csrc")

with open(os.path.join(ROOT, "tests", "golden", "ref_counts.json")) as _f:
    RECORDS = [r for r in json.load(_f)["records"] if r["order"] != "spiral" and not r.get("initial_situation")]


@pytest.fixture(scope="module")
def walk(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("compact") / "compact_search")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I" + CSRC, "-o", exe,
                    os.path.join(ROOT, "tests", "compact_search.cpp"), os.path.join(CSRC, "emp_compact.cpp"),
                    os.path.join(CSRC, "emp_model.cpp")], check=True)

    def run(puzzles, min_nw=1, split=0):
        text = "\n".join(f"{p.width} {p.height} {min_nw} {split} " + " ".join(str(c) for q in p.colors for c in q)
                         for p in puzzles)
        out = subprocess.run([exe], input=text + "\n", capture_output=True, text=True, check=True).stdout
        return [None if l == "none" else tuple(int(v) for v in l.split()) for l in out.splitlines()]
    return run


@pytest.mark.parametrize("min_nw,split", [(1, 0), (1, 7), (2, 0), (4, 50)])
def test_counts_equal_reference_build(walk, min_nw, split):
    recs = [r for r in RECORDS if r["nodes"] <= 200000]
    assert len(recs) > 50
    got = walk([Puzzle.from_csv(r["csv"]) for r in recs], min_nw, split)
    assert [g for g in got if g is None] == []
    for r, g in zip(recs, got):
        assert g == (r["nodes"], r["solutions"]), r["name"]


@pytest.mark.parametrize("colours", [1, 2, 3])
def test_few_colours_and_thin_boards(walk, colours):
    """Many identical and symmetric pieces, boards two and three wide."""
    rng = random.Random(colours)
    pzs = []
    while len(pzs) < 20:
        w, h = rng.randint(2, 5), rng.randint(2, 4)
        pz = generate(w, h, rng.randint(1, colours), rng.randint(1, colours), rng.randint(0, 1 << 30))
        if OraclePuzzle(w, h, pz.colors).estimate(200) < 1e5:
            pzs.append(pz)
    got = walk(pzs, split=5)
    assert sum(g is not None for g in got) >= 15
    for pz, g in zip(pzs, got):
        if g is not None:
            want, _ = OraclePuzzle(pz.width, pz.height, pz.colors).run()
            assert g == (want.nodes, want.solutions)


def test_wide_boards(walk):
    """Several words of centre slots: the first placements of boards whose trees are small."""
    pzs = [generate(9, 9, 8, 20, 1), generate(10, 10, 8, 21, 2), generate(12, 9, 9, 21, 3)]
    for pz, g in zip(pzs, walk(pzs, split=100)):
        want, _ = OraclePuzzle(pz.width, pz.height, pz.colors).run()
        assert g == (want.nodes, want.solutions)


def test_boards_without_compact_tables(walk):
    """More border pieces than the border space holds."""
    assert walk([generate(2, 40, 3, 3, 1)]) == [None]
