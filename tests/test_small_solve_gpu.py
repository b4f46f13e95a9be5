"""Small heads-up subgames, whose iterations run in one cooperative kernel
(k_small_solve), against the no-allocation entry point, which launches every
level and terminal kind by itself: the same sums in the same order, so every
output is equal bit for bit.  Full ranges of every street (135 to 147 blocks of
8 hands), iteration counts around a launch's 128, a session continued in parts,
and several solves at once from different threads."""
import ctypes
import threading

import numpy as np
import pytest

import street_solver_gpu as ssg
import workloads as wl
from test_zz_no_alloc import noalloc_solve

pytestmark = pytest.mark.gpu


def make(nb, bets, raises, hands=None, seed=1):
    rng = np.random.default_rng(seed)
    board = [int(c) for c in rng.permutation(52)[:nb]]
    h, w = wl.make_ranges(rng, board, 2, hands, zero_frac=0.1)
    cfg = dict(board=board, pot=100, stack=400, bet_sizes=bets, max_raises=raises, num_players=2, seed=seed)
    cfg["hands"], cfg["weights"] = h, w
    sg = wl.AbiSubgame(cfg, max_hands=ssg.SS_MAX_HANDS_WIDE)
    sg.set_leaf_values(wl.leaf_values_for(cfg, sg.num_leaves))
    return sg


def check(got, ref):
    for k in ("avg_strategies", "root_strategy", "root_ev"):
        assert np.array_equal(got[k], ref[k]), k


@pytest.mark.parametrize("nb,bets,raises,iterations", [
    (5, [0.5, 1.0], 2, 40), (5, [0.25, 0.5, 1.0, 2.0], 3, 12), (4, [0.33, 0.75], 2, 8), (3, [1.0], 2, 6),
])
def test_full_ranges(nb, bets, raises, iterations):
    sg = make(nb, bets, raises)
    rc, got = sg.solve(iterations)
    assert rc == 0, ssg.last_error(sg.lib)
    check(got, noalloc_solve(sg, iterations))
    sg.free()


@pytest.mark.parametrize("iterations", [1, 127, 128, 129, 300])
def test_iterations_around_a_launch(iterations):
    sg = make(5, [0.5, 1.0], 2, hands=30)
    rc, got = sg.solve(iterations)
    assert rc == 0, ssg.last_error(sg.lib)
    check(got, noalloc_solve(sg, iterations))
    sg.free()


def test_session_in_parts_and_reset():
    sg = make(4, [0.5, 1.0], 2, hands=120)
    ssg._session_api(sg.lib)
    sg.lib.ss_session_reset.argtypes = [ctypes.c_void_p]
    opts = ssg.SSSolveOptions(0, 10, -1.0, 50, 0)
    sess = ctypes.c_void_p()
    assert sg.lib.ss_session_create(ctypes.byref(sg.td), ctypes.byref(opts), ctypes.byref(sess)) == 0
    ref = noalloc_solve(sg, 20)
    for parts in ((20,), (3, 17), (1, 1, 18)):
        assert sg.lib.ss_session_reset(sess) == 0
        for n in parts:
            assert sg.lib.ss_session_run(sess, n) == 0
        out = ssg.SSOutput()
        assert sg.lib.ss_session_output(sess, ctypes.byref(out)) == 0
        check(wl.read_output(out, sg.nh), ref)
        sg.lib.ss_free_output(ctypes.byref(out))
    sg.lib.ss_session_destroy(sess)
    sg.free()


def test_solves_from_several_threads():
    subs = [make(5, [0.5, 1.0], 2, hands=n, seed=n) for n in (40, 300, 1081, 90)]
    refs = [noalloc_solve(sg, 150) for sg in subs]
    got, errors = [[] for _ in subs], []

    def work(i):
        for _ in range(3):
            rc, r = subs[i].solve(150)
            if rc != 0:
                errors.append(ssg.last_error(subs[i].lib))
                return
            got[i].append(r)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(subs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for i, ref in enumerate(refs):
        assert len(got[i]) == 3
        for r in got[i]:
            check(r, ref)
    for sg in subs:
        sg.free()
