"""A batch's terminal launches go side by side within one traverser's pass
only: traversers write the same value rows.  A player who makes no decision
(all in before the street) has no value or reach launches that would stand
between its terminals and the next traverser's; such trees come from a caller,
the library's builder makes none."""
import itertools
import json
import os
import shutil
import subprocess

import numpy as np
import pytest

import workloads as wl

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
TERM = 2


@pytest.fixture(scope="module")
def emul(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    out = str(tmp_path_factory.mktemp("runs") / "runs_emul")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "poker-solver_b200", "csrc"),
                    os.path.join(ROOT, "tests", "native", "runs_emul.cpp"), "-o", out], check=True)
    return out


@pytest.mark.parametrize("players", [1, 2, 3, 4])
def test_runs_hold_one_traverser(emul, players):
    for decides in range(1 << players):
        q = json.loads(subprocess.run([emul, str(players), str(decides)], capture_output=True, text=True,
                                      check=True).stdout)
        order = [t for _, type_, t, _ in q if type_ == TERM]
        assert order == sorted(order), (decides, q)   # traversers stay in order
        for run, launches in itertools.groupby(q, key=lambda x: x[0]):
            launches = list(launches)
            if launches[0][1] == TERM:
                assert len({t for _, _, t, _ in launches}) == 1 and len(launches) == 3, (decides, q)
                weights = [w for _, _, _, w in launches]
                assert weights == sorted(weights)
            else:
                assert len(launches) == 1


def subgame(name, seed, nh, **over):
    """A three-player subgame whose player 0 makes no decision: its nodes are
    player 1's."""
    cfg = wl.config(name, seed=seed, num_players=3, **over)
    cfg["hands"], cfg["weights"] = wl.make_ranges(np.random.default_rng(seed), cfg["board"], 3, nh)
    sg = wl.AbiSubgame(cfg, max_hands=200)
    sg.set_leaf_values(wl.leaf_values_for(cfg, sg.num_leaves))
    for i in range(sg.td.num_nodes):
        n = sg.td.nodes[i]
        if n.type == 0 and n.player == 0:
            n.player = 1
    return sg


@pytest.mark.gpu
def test_batch_of_trees_with_a_player_without_decisions():
    subs = [subgame("river6", 81, 40, bet_sizes=[1.0], max_raises=1), subgame("turn3", 82, 30, bet_sizes=[0.75], max_raises=1),
            subgame("river6", 83, 70, bet_sizes=[0.5, 1.0], max_raises=1)]
    alone = []
    for sg in subs:
        rc, r = sg.solve(23)
        assert rc == 0
        alone.append(r)
    for mix in ([0], [1], [0, 1, 2]):
        rc, together = wl.batch_solve([subs[i] for i in mix], 23, graph_iterations=10)
        assert rc == 0, wl.ssg.last_error(subs[0].lib)
        for i, r in zip(mix, together):
            for k in ("root_strategy", "root_ev", "avg_strategies", "avg_node_ids"):
                assert np.array_equal(r[k], alone[i][k]), (mix, i, k)
    for sg in subs:
        sg.free()
