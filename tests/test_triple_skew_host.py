"""Host check of the three-opponent mass where little of the product of the
ranges is left (poker-solver_b200/csrc/ss_triple.cuh, compiled with g++): the
third opponent's weight lies on hands that every traverser hand blocks, down
to 1e-16 elsewhere.

The contraction's error is below 1e-13 of the product of the ranges' sums (the
bound of test_triple_host.py), and masses up to 1e-6 of it are summed again
hand by hand of the third opponent, so a mass is right to 1e-13 / 1e-6 = 1e-7
of itself above that bound; below it every term is a two-opponent mass over
U(0, 1) ranges, right to better than that."""
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
    out = str(tmp_path_factory.mktemp("skew") / "triple_skew")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "poker-solver_b200", "csrc"),
                    os.path.join(ROOT, "tests", "native", "triple_skew.cpp"), "-o", out], check=True)
    return out


@pytest.mark.parametrize("repeat", [0, 1])
@pytest.mark.parametrize("rest", ["1", "1e-4", "1e-6", "1e-8", "1e-12", "1e-16", "0"])
@pytest.mark.parametrize("deck,hands", [(48, 120), (47, 90), (10, 40)])
def test_small_masses_keep_their_digits(emul, deck, hands, rest, repeat):
    res = json.loads(subprocess.run([emul, "7", str(deck), str(hands), rest, "2", str(repeat)], capture_output=True,
                                    text=True, check=True).stdout)
    assert res["worst"] <= 1e-7, res
    assert res["zero_bad"] == 0, res
