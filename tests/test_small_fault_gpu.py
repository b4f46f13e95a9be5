"""A grid-wide wait of a session's iterations that runs out (its limit set to
0: a block that is not the last to arrive gives up at once) is reported by
every call that waits for that session or reads its state until the state is
reset, and by no other session."""
import ctypes

import numpy as np
import pytest

import street_solver_gpu as ssg
import workloads as wl
from test_small_solve_gpu import check, make

pytestmark = pytest.mark.gpu
LIMIT = 4 << 20


def session(sg):
    lib = sg.lib
    ssg._session_api(lib)
    vp = ctypes.c_void_p
    lib.ss_session_reset.argtypes = [vp]
    lib.ss_session_synchronize.argtypes = [vp]
    lib.ss_session_exploitability.argtypes = [vp] + 5 * [ctypes.c_void_p]
    lib.ss_session_profile.argtypes = [vp, vp]
    lib.ss_session_set_wait_limit.argtypes = [vp, ctypes.c_uint]
    opts = ssg.SSSolveOptions(0, 10, -1.0, 50, 0)
    s = vp()
    assert lib.ss_session_create(ctypes.byref(sg.td), ctypes.byref(opts), ctypes.byref(s)) == 0
    return s


def output(sg, s):
    out = ssg.SSOutput()
    rc = sg.lib.ss_session_output(s, ctypes.byref(out))
    if rc != 0:
        return rc, None
    r = wl.read_output(out, sg.nh)
    sg.lib.ss_free_output(ctypes.byref(out))
    return 0, r


@pytest.mark.parametrize("nb,iterations", [(5, 3), (4, 200)])
def test_a_lost_wait_stays_with_its_session(nb, iterations):
    sg = make(nb, [0.5, 1.0], 2, hands=90)
    lib = sg.lib
    a, b = session(sg), session(sg)
    assert lib.ss_session_set_wait_limit(a, 0) == 0
    assert lib.ss_session_run(a, iterations) == 0       # queued
    assert lib.ss_session_run(b, iterations) == 0
    rc, got = output(sg, b)                              # the other session first
    assert rc == 0, ssg.last_error(lib)
    pct = ctypes.c_double()
    w = np.ones(len(sg.H[0]))
    keep = w.copy()
    hands = np.ascontiguousarray(sg.H[0][:90], np.int32)
    prof = ctypes.create_string_buffer(4096)
    reads = [
        lambda: lib.ss_session_synchronize(a),
        lambda: output(sg, a)[0],
        lambda: lib.ss_session_exploitability(a, ctypes.byref(pct), None, None, None, None),
        lambda: lib.ss_session_narrow(a, 0, -1, 1, len(hands), hands.ctypes.data_as(ctypes.POINTER(ctypes.c_int)),
                                      w.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), None),
        lambda: lib.ss_session_profile(a, prof),
        lambda: output(sg, a)[0],
        lambda: lib.ss_session_run(a, 1),
    ]
    for first in range(len(reads) - 1):                 # any of them may be the first to look
        for r in reads[first:] + reads[:first]:
            assert r() == -2
            assert "wait" in ssg.last_error(lib)
        assert np.array_equal(w, keep)
        assert lib.ss_session_reset(a) == 0
        assert lib.ss_session_run(a, iterations) == 0
    assert lib.ss_session_synchronize(a) == -2
    assert lib.ss_session_set_wait_limit(a, LIMIT) == 0
    assert lib.ss_session_reset(a) == 0
    assert lib.ss_session_run(a, iterations) == 0
    rc, again = output(sg, a)
    assert rc == 0, ssg.last_error(lib)
    check(again, got)
    assert lib.ss_session_exploitability(b, ctypes.byref(pct), None, None, None, None) == 0
    lib.ss_session_destroy(a)
    lib.ss_session_destroy(b)
    sg.free()
