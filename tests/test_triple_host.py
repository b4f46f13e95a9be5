"""Host check of the three-opponent mass by contraction (the block phases of
poker-solver_b200/csrc/ss_triple.cuh, compiled with g++): every traverser
hand against enumeration of the pairwise disjoint opponent tuples, on flop,
turn and river decks and tiny ones where most hands have no tuple, with
zeroed weights, an opponent without reach and a third range that repeats
combos.  The mass is a sum of some 20 terms of at most a few products of the
ranges' sums, each rounded a few hundred times: 1e-13 of that product."""
import json
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def emul(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    out = str(tmp_path_factory.mktemp("triple") / "triple_emul")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "poker-solver_b200", "csrc"),
                    os.path.join(ROOT, "tests", "native", "triple_emul.cpp"), "-o", out], check=True)
    return out


@pytest.mark.parametrize("args", [
    (1, 48, 160, 0.3, 0), (2, 47, 130, 0.0, 0), (3, 49, 100, 0.6, 0), (4, 48, 90, 0.3, 1), (5, 52, 60, 0.0, 0),
    (6, 6, 15, 0.0, 0), (7, 7, 16, 0.4, 0), (8, 8, 20, 0.2, 1), (9, 10, 16, 0.9, 0), (10, 48, 40, 0.3, 0, 1),
    (11, 46, 64, 0.95, 1),
])
def test_contraction_equals_enumeration(emul, args):
    res = json.loads(subprocess.run([emul] + [str(a) for a in args], capture_output=True, text=True, check=True).stdout)
    assert res["worst"] <= 1e-13, res
    assert res["zero_bad"] == 0, res
