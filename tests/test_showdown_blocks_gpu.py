"""Two-way showdowns in small and in large blocks (launches of more than 296 and
of up to 296 of them) give the same bits: a batch whose launches hold just as
many, more and far more, and a river with thousands, against solves in the
other form (alone, where small subgames take k_small_solve, and member by
member), repeated combos included."""
import numpy as np
import pytest

import street_solver_gpu as ssg
import workloads as wl
from test_parity_gpu import oracle_pair, solve, strict

pytestmark = pytest.mark.gpu


def river(seed, hands, bets, raises, repeat=False, pot=100, stack=400):
    rng = np.random.default_rng(seed)
    board = [int(c) for c in rng.permutation(52)[:5]]
    h, w = wl.make_ranges(rng, board, 2, hands, zero_frac=0.1)
    if repeat:   # some combos twice, in either player's range
        h = [np.concatenate([x, x[:5]]) for x in h]
        w = [np.concatenate([x, x[5:10]]) for x in w]
    cfg = dict(board=board, pot=pot, stack=stack, bet_sizes=bets, max_raises=raises, num_players=2, seed=seed, hands=h,
               weights=w)
    return wl.AbiSubgame(cfg, max_hands=ssg.SS_MAX_HANDS_WIDE)


def showdowns(sg):
    return sum(sg.td.nodes[i].type == 2 for i in range(sg.td.num_nodes))


@pytest.mark.parametrize("hands,repeat", [(40, False), (None, False), (40, True)])
def test_batches_around_the_line(hands, repeat):
    first = river(1, hands, [0.5, 1.0], 2, repeat)
    per = showdowns(first)
    fit = 296 // per
    subs = [first] + [river(s, hands, [0.5, 1.0], 2, repeat) for s in range(2, fit + 2)] + \
        [river(s, hands, [0.5, 1.0], 2, repeat) for s in range(100, 100 + 2 * fit)]
    assert all(showdowns(sg) == per for sg in subs)
    assert fit * per <= 296 < (fit + 1) * per
    alone = []
    for sg in subs:
        rc, r = sg.solve(9)
        assert rc == 0, ssg.last_error(sg.lib)
        alone.append(r)
    for n in (fit, fit + 1, len(subs)):
        rc, got = wl.batch_solve(subs[:n], 9)
        assert rc == 0, ssg.last_error(first.lib)
        for r, a in zip(got, alone):
            for k in ("avg_strategies", "root_strategy", "root_ev"):
                assert np.array_equal(r[k], a[k]), (n, k)
    # the FP64 form: the members' exploitabilities in one launch and alone
    rc, many = wl.batch_solve(subs, 9, target=1e-6, check_every=9)
    assert rc == 0
    for sg, r in zip(subs[:3], many):
        rc, one = wl.batch_solve([sg], 9, target=1e-6, check_every=9)
        assert rc == 0
        assert one[0]["stats"]["exploitability_pct"] == r["stats"]["exploitability_pct"]
    for sg in subs:
        sg.free()


def test_a_river_with_thousands_against_the_oracle(oracle):
    cfg = wl.config("hu_river", seed=7, num_hands=20, bet_sizes=[0.25, 0.5, 0.75, 1.0, 1.5], max_raises=5, stack=5000)
    ours, lv = solve(cfg, 3)
    r32, _ = oracle_pair(oracle, cfg, 3, lv)
    strict(ours, r32)
