"""Small heads-up sessions beside others: the route of a call (one cooperative
kernel, or kernel by kernel where the device is full of others' grids) does not
show in the results.  Sessions keep long runs in flight on their own streams
while one session is stepped, in calls of every length, across both routes; all
of them end with what the no-allocation entry point gives, bit for bit.  Which
route a call took shows in a wait limit of 0: only the cooperative kernel waits."""
import ctypes
import threading

import pytest

import street_solver_gpu as ssg
from test_small_fault_gpu import LIMIT, output, session
from test_small_solve_gpu import check, make
from test_zz_no_alloc import noalloc_solve

pytestmark = pytest.mark.gpu

# a river and two turns: tree passes, and above the line level by level
CASES = [(5, [0.5, 1.0], 2, None), (4, [0.5, 1.0], 2, 300), (4, [0.33, 0.75, 1.5], 3, None)]


def crowd(n=8):
    """Sessions that fill the device several times over, and their subgame."""
    sg = make(5, [0.5, 1.0], 2)
    return sg, [session(sg) for _ in range(n)]


@pytest.mark.parametrize("nb,bets,raises,hands", CASES)
def test_results_do_not_depend_on_the_route(nb, bets, raises, hands):
    big, others = crowd()
    lib = big.lib
    sg = make(nb, bets, raises, hands=hands, seed=5)
    s = session(sg)
    alone = session(sg)
    parts = (1, 2, 16, 30, 1, 50)
    ref = noalloc_solve(sg, sum(parts))
    for _ in range(2):                       # the second time with the graphs of the first
        for i, n in enumerate(parts):
            for o in others:                 # in flight beside every other call
                if i % 2 == 0:
                    assert lib.ss_session_run(o, 128) == 0
            assert lib.ss_session_run(s, n) == 0
            assert lib.ss_session_run(alone, n) == 0
        rc, got = output(sg, s)
        assert rc == 0, ssg.last_error(lib)
        check(got, ref)
        rc, got = output(sg, alone)
        assert rc == 0, ssg.last_error(lib)
        check(got, ref)
        assert lib.ss_session_reset(s) == 0 and lib.ss_session_reset(alone) == 0
    for x in others + [s, alone]:
        lib.ss_session_destroy(x)
    big.free()
    sg.free()


def test_a_crowded_session_is_launched_kernel_by_kernel():
    big, others = crowd(10)
    lib = big.lib
    sg = make(5, [0.5, 1.0], 2, seed=6)
    s = session(sg)
    assert lib.ss_session_set_wait_limit(s, 0) == 0
    assert lib.ss_session_run(s, 2) == 0             # alone: the cooperative kernel, which gives up
    assert output(sg, s)[0] == -2
    for _ in range(4):                               # (the mean over the calls follows)
        for o in others:
            assert lib.ss_session_run(o, 1000) == 0
    assert lib.ss_session_reset(s) == 0
    assert lib.ss_session_run(s, 5) == 0             # kernel by kernel: nothing to give up
    rc, got = output(sg, s)
    assert rc == 0, ssg.last_error(lib)
    check(got, noalloc_solve(sg, 5))
    for o in others:
        assert lib.ss_session_synchronize(o) == 0
    assert lib.ss_session_set_wait_limit(s, LIMIT) == 0
    for x in others + [s]:
        lib.ss_session_destroy(x)
    big.free()
    sg.free()


def test_sessions_come_and_go_on_many_threads():
    subs = [make(5, [0.5, 1.0], 2, hands=h, seed=20 + i) for i, h in enumerate((40, 300, 1081, 90, 700, 1081, 200, 500))]
    refs = [noalloc_solve(sg, 60) for sg in subs]
    errors = []

    def work(i):
        for _ in range(6):
            rc, r = subs[i].solve(60)
            if rc != 0:
                errors.append((i, ssg.last_error(subs[i].lib)))
                return
            try:
                check(r, refs[i])
            except AssertionError as e:
                errors.append((i, str(e)))
                return

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(subs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for sg in subs:
        sg.free()
