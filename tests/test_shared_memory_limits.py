"""The shared-memory limit of a kernel is one attribute for all host threads,
so every call sets it to the same value: the largest launch's, never this
launch's size (which another thread could lower under a larger launch)."""
import glob
import os
import re
import threading

import numpy as np
import pytest

import street_solver_gpu as ssg
import workloads as wl

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_limits_do_not_depend_on_the_launch():
    seen = 0
    for path in glob.glob(os.path.join(ROOT, "poker-solver_b200", "csrc", "*.cu*")):
        src = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"cudaFuncSetAttribute\(\s*([\w<>]+),\s*cudaFuncAttributeMaxDynamicSharedMemorySize,", src):
            i, depth = m.end(), 1
            while depth:
                depth += {"(": 1, ")": -1}.get(src[i], 0)
                i += 1
            limit = src[m.end():i - 1]
            assert not re.search(r"\bsm\b|\bc\.|\bn_|\bspan\b|\.bytes", limit), (os.path.basename(path), m.group(1), limit)
            seen += 1
    assert seen >= 10


@pytest.mark.gpu
def test_three_way_showdowns_of_different_sizes_at_once():
    subs = []
    for i, n in enumerate((12, 60, 250, 700)):
        cfg = wl.config("river6", seed=90 + i, num_players=3, bet_sizes=[1.0], max_raises=1)
        cfg["hands"], cfg["weights"] = wl.make_ranges(np.random.default_rng(90 + i), cfg["board"], 3, n)
        subs.append(wl.AbiSubgame(cfg, max_hands=ssg.SS_MAX_HANDS_WIDE))
    alone = []
    for sg in subs:
        rc, r = sg.solve(12)
        assert rc == 0
        alone.append(r)
    errors = []

    def work(i):
        for _ in range(12):
            rc, r = subs[i].solve(12)
            if rc != 0:
                errors.append((i, rc, ssg.last_error(subs[i].lib)))
            elif not all(np.array_equal(r[k], alone[i][k]) for k in ("root_strategy", "root_ev", "avg_strategies")):
                errors.append((i, "differs"))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(subs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for sg in subs:
        sg.free()
