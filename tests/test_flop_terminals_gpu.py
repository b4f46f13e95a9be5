"""Every node's value of the multi-street solver after one iteration (uniform
play) against the FP64 restatement, where the showdown tables and the
terminal sums can go wrong: one hand, hand counts around a warp, unequal
ranges, ranges that touch the flop, repeat a combo or hold zero weights.
After one iteration nothing has been amplified: a value is a sum over at most
11 tree levels of at most 49 FP32 additions each, 3e-5 of its terms, within
the 1e-4 of the largest value that the other tests use; a terminal value that
is exactly 0 (no compatible hand wins or loses) is exactly 0."""
import numpy as np
import pytest

import flop_solve as fsm
import street_solver_gpu as ssg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed,n0,n1,zero,touch,repeat", [
    (1, 1, 1, 0.0, False, False),
    (2, 31, 33, 0.0, False, False),
    (3, 32, 7, 0.5, True, False),
    (4, 20, 36, 0.2, True, True),
])
def test_values_after_one_iteration(seed, n0, n1, zero, touch, repeat):
    from oracle.oracle import FlopOracle
    rng = np.random.default_rng(seed)
    flop = [int(c) for c in rng.permutation(52)[:3]]
    combos = [(a, b) for a in range(52) for b in range(a + 1, 52)
              if touch or (a not in flop and b not in flop)]
    hands, weights = [], []
    for n in (n0, n1):
        h = np.array([combos[i] for i in rng.choice(len(combos), n, replace=False)], np.int32)
        if repeat:
            h[-3:] = h[:3]
        w = rng.uniform(0.1, 1.0, n).astype(np.float32)
        w[rng.random(n) < zero] = 0.0
        hands.append(h)
        weights.append(w)
    sg = fsm.FlopSubgame(ssg.load_library(200), flop, 1000, 5000, [0.75], hands, weights)
    got = sg.solve(1, extract=True)
    nodes, ch, _, nd, _, _ = fsm.tree_arrays(sg.td)
    depth = sg.td.max_depth
    sg.free()
    H, W = np.zeros((2, 200, 2), np.int32), np.zeros((2, 200), np.float32)
    for p in range(2):
        H[p, :len(hands[p])], W[p, :len(hands[p])] = hands[p], weights[p]
    ref = FlopOracle().solve(nodes, ch, nd, depth, H, W, np.array([n0, n1], np.int32), 1, "f64")
    a, b = got["all_cfv"], ref["all_cfv"]
    scale = max(np.abs(b).max(), 1e-30)
    assert np.abs(a - b).max() <= 1e-4 * scale
    term = (nodes[:, 0] == fsm.NODE_FOLD) | (nodes[:, 0] == fsm.NODE_SHOWDOWN)
    assert np.all(a[term][b[term] == 0] == 0)
