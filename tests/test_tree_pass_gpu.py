"""The one-launch pass over a player's small tree levels (k_tree) against the
form with a launch per level (k_cfv, k_reach), which the no-allocation entry
point runs: both add and update in the same order, so every output is equal
bit for bit.  Hand counts around the 8-hand blocks, one to five actions plus
all-in, long frontiers (summed in four interleaved chains), levels on both
sides of the pass's bound, frozen actions, repeated combos."""
import numpy as np
import pytest

import workloads as wl
from test_zz_no_alloc import noalloc_solve

pytestmark = pytest.mark.gpu

CASES = [
    # players, board cards, bets, raises, hands, iterations
    (2, 5, [1.0], 1, 1, 9),
    (2, 5, [0.5, 1.0], 2, 7, 25),
    (2, 5, [0.33, 0.75, 1.5], 3, 8, 12),
    (2, 5, [0.25, 0.5, 1.0, 2.0], 3, 9, 12),
    (2, 5, [0.2, 0.4, 0.6, 0.8, 1.0], 2, 33, 11),     # 8 actions at the facing nodes
    (2, 4, [0.33, 0.75, 1.5], 3, 63, 8),               # 188 items in one level: past the bound
    (2, 3, [0.5], 1, 200, 6),
    (3, 5, [0.5, 1.0], 2, 65, 6),
    (3, 4, [0.5], 2, 31, 5),                           # long frontiers
    (4, 5, [0.5], 2, 17, 3),
]


def make(case, frozen=False, dup=False):
    players, nb, bets, raises, hands, _ = case
    rng = np.random.default_rng(hands)
    board = [int(c) for c in rng.permutation(52)[:nb]]
    h, w = wl.make_ranges(rng, board, players, hands, zero_frac=0.2)
    if dup:
        h[1][-1] = h[1][0]
    cfg = dict(board=board, pot=100, stack=400, bet_sizes=bets, max_raises=raises, num_players=players, seed=hands)
    cfg["hands"], cfg["weights"] = h, w
    sg = wl.AbiSubgame(cfg)
    sg.set_leaf_values(wl.leaf_values_for(cfg, sg.num_leaves))
    if frozen:
        nodes = sg.tree_arrays()[0]
        fr = np.where((nodes[:, 0] == 0) & (np.arange(len(nodes)) % 3 == 0), nodes[:, 2] - 1, -1).astype(np.int32)
        sg.set_frozen(fr)
    return sg


def equal_outputs(sg, iterations):
    ref = noalloc_solve(sg, iterations)
    rc, got = sg.solve(iterations)
    assert rc == 0, wl.ssg.last_error(sg.lib)
    for k in ("avg_strategies", "root_strategy", "root_ev"):
        assert np.array_equal(got[k], ref[k]), k


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"{c[0]}p{c[1]}b{len(c[2])}x{c[3]}h{c[4]}")
def test_tree_pass_equals_level_launches(case):
    sg = make(case)
    equal_outputs(sg, case[-1])
    sg.free()


@pytest.mark.parametrize("frozen,dup", [(True, False), (False, True)])
def test_tree_pass_frozen_and_repeated_combos(frozen, dup):
    for case in (CASES[2], CASES[7]):
        sg = make(case, frozen, dup)
        equal_outputs(sg, case[-1])
        sg.free()
