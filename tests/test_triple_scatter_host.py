"""Host check of the three-opponent matrices (poker-solver_b200/csrc/ss_triple.cuh):
written hand by hand, as k_term_cr3 does, and looked up pair by pair they are
the same bits, nonzero cells' masks included -- flop, turn, river and tiny decks,
ranges of one hand and of every combo, zero weights, blocked hands and a third
range that repeats combos."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def emul(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    out = str(tmp_path_factory.mktemp("scatter") / "triple_scatter")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "poker-solver_b200", "csrc"),
                    os.path.join(ROOT, "tests", "native", "triple_scatter.cpp"), "-o", out], check=True)
    return out


@pytest.mark.parametrize("repeat", [0, 1])
@pytest.mark.parametrize("deck,hands,zero", [(48, 1, 0), (48, 60, 0.3), (47, 1081, 0), (49, 1176, 0.5), (52, 1326, 0),
                                            (6, 15, 0.2), (48, 100, 1)])
def test_scatter_equals_lookup(emul, deck, hands, zero, repeat):
    r = subprocess.run([emul, "3", str(deck), str(hands), str(zero), str(repeat)], capture_output=True, text=True,
                       check=True)
    assert int(r.stdout) == 0
