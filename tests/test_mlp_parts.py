"""A training run sizes its workspace once, for its batch, and its last minibatch is smaller: the
partial sums of any smaller row count fit (on the CPU, from the layout the launches use), and an
epoch whose last minibatch needs more of them than a whole batch has the float64 oracle's loss."""
from __future__ import annotations

import ctypes
import os
import subprocess

import numpy as np
import pytest

from edge_matching_puzzle_b200 import native
from edge_matching_puzzle_b200.puzzle import generate, row_major_order
from oracle import mlp_oracle
from oracle.oracle import OraclePuzzle

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_smaller_row_counts_fit(tmp_path):
    exe = str(tmp_path / "mlp_parts")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I/usr/local/cuda/include",
                    "-I" + os.path.join(ROOT, "edge_matching_puzzle_b200", "csrc"), "-o", exe,
                    os.path.join(ROOT, "tests", "mlp_parts.cpp")], check=True)
    assert subprocess.run([exe], capture_output=True, text=True, check=True).stdout == "fits\n"


def _solved(seed):
    """A 6x6 board without identical pieces and its first solution, as transitions a level."""
    pz = generate(6, 6, 4, 8, seed)
    op = OraclePuzzle(6, 6, pz.colors)
    r, _ = op.run(node_limit=3_000_000)
    if op.has_identical or not r.solutions:
        return None
    kinds = {op.piece_of(k, i): (k, i) for k in range(3) for i in range(op.nb_kind(k))}
    board = list(r.first_board)[:36]
    return pz, op, board, [(kinds[v >> 2][1] << 2) | (v & 3) for v in board]


def _samples(pz, op, board, path):
    """Per level after the first: every candidate that the search tries after what was placed
    before (a trial takes out what its identical mask clears), and whether it is the solution's."""
    col = pz.colors
    members = [[op.piece_of(k, i) for i in range(op.nb_kind(k))] for k in range(3)]
    out = []
    for l in range(1, 35):
        x, y = l % 6, l // 6
        used = {v >> 2 for v in board[:l]}
        kind = (x in (0, 5)) + (y in (0, 5))
        row = []
        for i, p in enumerate(members[kind]):
            for o in range(0, 4, op.orientation_step(p)):  # the turns the reference tries
                side = [col[p][(s + o) % 4] for s in range(4)]
                facing = lambda pos, s: col[board[pos] >> 2][(s + (board[pos] & 3)) % 4]
                ok = (side[0] == 0) == (y == 0) and (side[1] == 0) == (x == 5) and (side[2] == 0) == (y == 5) and \
                    (side[3] == 0) == (x == 0) and (y == 0 or side[0] == facing(l - 6, 2)) and \
                    (x == 0 or side[3] == facing(l - 1, 1))
                if ok and p not in used:
                    row.append((i << 2) | o)
        tried = []
        while row:
            tried.append(row[0])
            keep = op.identical_mask(kind, row[0])
            row = [t for t in row[1:] if keep[t >> 6] >> (t & 63) & 1]
        out.append([(mlp_oracle.features(6, 6, col, row_major_order(6, 6), members, path[:l], t), t == path[l])
                    for t in tried])
    return out


class _SplitMix:
    def __init__(self, state):
        self.s = state

    def __call__(self):
        m = (1 << 64) - 1
        self.s = (self.s + 0x9E3779B97F4A7C15) & m
        z = self.s
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & m
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & m
        return z ^ (z >> 31)


@pytest.mark.gpu
def test_epoch_with_a_smaller_last_minibatch_matches_fp64_oracle():
    """The loss that the run reports lies behind the partial sums in the workspace, and each
    gradient is divided by its weights' sum beside it.  Tolerance: the f32 losses are off by 1e-6; a
    gradient too small for its sign to be sure (1e-7) turns Adam's first step of a parameter by
    up to 2 lr, which moves the second loss by at most 2e-10 a parameter, 4e-5 for all.  (The parameters
    themselves cannot be compared closer than such a step, 2 lr.)"""
    solved, seed, total = [], 0, 0
    while total < 4049:
        s = _solved(seed)
        seed += 1
        if s:
            solved.append(s + (_samples(*s),))
            total += sum(len(r) for r in solved[-1][-1])
    batch, lr = total - 2000, 1e-3
    assert 2049 <= batch <= 2160
    rows = [q for l in range(34) for s in solved for q in s[-1][l]]  # by level, then by puzzle
    x = np.array([q[0] for q in rows])
    y = np.array([float(q[1]) for q in rows])
    w = np.where(y > 0.5, (len(y) - y.sum()) / y.sum(), 1.0)
    handles = [native.NativePuzzle(6, 6, s[0].colors) for s in solved]
    m = native.Mlp(seed=9)
    p = m.params().astype(np.float64)
    start = p.copy()
    boards = [s[2] + [0xFFFFFFFF] * 220 for s in solved]
    rep = m.train(handles, boards, epochs=1, batch=batch, learning_rate=lr, seed=1)
    assert rep.samples == total
    order, rng = list(range(total)), _SplitMix(1)
    for i in range(total - 1, 0, -1):
        j = rng() % (i + 1)
        order[i], order[j] = order[j], order[i]
    m1, m2, losses = np.zeros_like(p), np.zeros_like(p), 0.0
    for step, part in enumerate((order[:batch], order[batch:]), 1):
        loss, g = mlp_oracle.loss_grad(p, x[part], y[part], w[part])
        losses += loss * w[part].sum()
        m1, m2 = 0.9 * m1 + 0.1 * g, 0.999 * m2 + 0.001 * g * g
        p -= lr * (m1 / (1 - 0.9 ** step)) / (np.sqrt(m2 / (1 - 0.999 ** step)) + 1e-8)
    assert abs(rep.first_loss - losses / w.sum()) <= 1e-4
    assert np.max(np.abs(m.params() - start)) <= 2.2 * lr  # two steps of at most lr (1 + 0.053)
