"""Iterations launched one by one, or as graphs of one or several, give the
same bits however a run is cut: against the no-allocation entry point, which
launches everything in order.  Totals on both sides of the rules (16
iterations without a graph, graphs of 1, 2 and 3 from 17, 128 and 384 on)."""
import ctypes

import numpy as np
import pytest

import workloads as wl
from test_tree_pass_gpu import make
from test_zz_no_alloc import noalloc_solve

pytestmark = pytest.mark.gpu

CASE = (3, 5, [1.0], 1, 9, 0)   # not one launch: three players


@pytest.mark.parametrize("runs,most", [
    ([16], 10), ([17], 10), ([1, 15, 1, 1], 10), ([18, 2, 3], 10), ([127], 10), ([128, 1, 5], 10),
    ([100, 100, 190], 10), ([390], 2), ([40], 1),
])
def test_cuts_of_a_run(runs, most):
    sg = make(CASE)
    ref = noalloc_solve(sg, sum(runs))
    lib = sg.lib
    wl.ssg._session_api(lib)
    opts = wl.ssg.SSSolveOptions(0, most, -1.0, 50, 0)
    sess, out = ctypes.c_void_p(), wl.ssg.SSOutput()
    assert lib.ss_session_create(ctypes.byref(sg.td), ctypes.byref(opts), ctypes.byref(sess)) == 0
    try:
        for n in runs:
            assert lib.ss_session_run(sess, n) == 0, wl.ssg.last_error(lib)
        assert lib.ss_session_output(sess, ctypes.byref(out)) == 0, wl.ssg.last_error(lib)
        n = out.num_avg_nodes * wl.ssg.SS_MAX_ACTIONS * out.max_hands
        avg = np.ctypeslib.as_array(out.avg_strategies, shape=(n,)).copy()
        rs = np.ctypeslib.as_array(out.root_strategy, shape=(out.root_num_actions * CASE[4],)).copy()
        lib.ss_free_output(ctypes.byref(out))
    finally:
        lib.ss_session_destroy(sess)
    assert np.array_equal(avg, np.asarray(ref["avg_strategies"]).ravel())
    assert np.array_equal(rs, np.asarray(ref["root_strategy"]).ravel())
    sg.free()


@pytest.mark.parametrize("iterations,most", [(1, 10), (40, 10), (150, 10), (390, 10), (390, 2)])
def test_batches_of_any_length(iterations, most):
    """Several players and kinds of terminals side by side, over graphs of 1 to
    3 iterations and what is left over."""
    subs = [make(c) for c in ((3, 5, [1.0], 1, 9, 0), (2, 5, [0.5, 1.0], 1, 40, 0), (4, 5, [1.0], 1, 17, 0),
                              (2, 4, [1.0], 1, 33, 0))]
    refs = [noalloc_solve(sg, iterations) for sg in subs]
    rc, got = wl.batch_solve(subs, iterations, graph_iterations=most)
    assert rc == 0, wl.ssg.last_error(subs[0].lib)
    for ref, r in zip(refs, got):
        for k in ("avg_strategies", "root_strategy", "root_ev"):
            assert np.array_equal(r[k], ref[k]), k
    for sg in subs:
        sg.free()
