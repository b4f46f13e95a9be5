"""Staged copies of large host buffers: continuation values whose bytes lie
around the staging bound (4 MiB), the piece size (1 MiB) and the threads'
shares, against the same rows from calls small enough for the plain copy; a
profile large enough to be staged up against the same profile solved for in
parts is covered by the full-size tests."""
import numpy as np
import pytest

import leaf_values as lv

pytestmark = pytest.mark.gpu

HANDS = 64
ROW = 4 * 16 * 2 * HANDS      # bytes per leaf descriptor: 16 profiles x 2 players x 64 hands
MIB = 1 << 20


@pytest.mark.parametrize("nbytes", [4 * MIB - ROW, 4 * MIB, 4 * MIB + ROW, 8 * MIB + ROW, 11 * MIB + 3 * ROW,
                                    33 * MIB + ROW])
def test_staged_values_equal_plain_ones(nbytes):
    rng = np.random.default_rng(7)
    board = [0, 13, 26, 39]
    deck = [c for c in range(52) if c not in board]
    combos = [(a, b, 1.0) for i, a in enumerate(deck) for b in deck[i + 1:]]
    ranges = [[combos[i] for i in np.sort(rng.choice(len(combos), HANDS, replace=False))] for _ in range(2)]
    n = nbytes // ROW
    infos = [lv.LeafInfo(i, 100 + i, (0, 0)) for i in range(n)]
    got = lv.compute_turn_leaf_values(board, infos, HANDS, 100, player_hands=ranges)
    assert got.nbytes == n * ROW
    step = 400
    for at in range(0, n, step):
        part = [lv.LeafInfo(i, 100 + at + i, (0, 0)) for i in range(min(step, n - at))]
        small = lv.compute_turn_leaf_values(board, part, HANDS, 100, player_hands=ranges)
        assert np.array_equal(got[at * 16:at * 16 + len(small)], small)
