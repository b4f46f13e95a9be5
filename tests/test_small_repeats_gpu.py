"""Small heads-up rivers whose ranges repeat combos.  With folds the terminals
of such ranges are of a kind that k_small_solve does not serve; a caller's tree
without folds (every one of them made a showdown here) is served, and adds the
repeated hands up position by position.  Against the no-allocation entry point,
bit for bit (a combo is held twice, so no order of additions is left open)."""
import ctypes

import numpy as np
import pytest

import street_solver_gpu as ssg
import workloads as wl
from test_small_fault_gpu import output, session
from test_small_solve_gpu import check
from test_zz_no_alloc import noalloc_solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hands,who", [(40, (0,)), (90, (1,)), (300, (0, 1)), (1000, (0, 1))])
def test_repeated_combos_without_folds(hands, who):
    rng = np.random.default_rng(hands)
    board = [int(c) for c in rng.permutation(52)[:5]]
    h, w = wl.make_ranges(rng, board, 2, hands, zero_frac=0.2)
    for p in who:
        n = hands // 8
        h[p] = np.concatenate([h[p], h[p][:n]])
        w[p] = np.concatenate([w[p], rng.uniform(0.0, 1.0, n).astype(np.float32)])
    cfg = dict(board=board, pot=100, stack=400, bet_sizes=[0.5, 1.0], max_raises=2, num_players=2, seed=hands, hands=h,
               weights=w)
    sg = wl.AbiSubgame(cfg, max_hands=ssg.SS_MAX_HANDS_WIDE)
    for i in range(sg.td.num_nodes):
        n = sg.td.nodes[i]
        if n.type == 1:
            n.type, n.player, n.num_players = 2, -1, 2
            n.active_players[0], n.active_players[1] = 1, 1
    rc, got = sg.solve(20)
    assert rc == 0, ssg.last_error(sg.lib)
    check(got, noalloc_solve(sg, 20))
    # the cooperative kernel ran it: only its waits can run out
    s = session(sg)
    assert sg.lib.ss_session_set_wait_limit(s, 0) == 0
    assert sg.lib.ss_session_run(s, 3) == 0
    assert output(sg, s)[0] == -2
    sg.lib.ss_session_destroy(s)
    sg.free()
