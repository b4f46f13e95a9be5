"""Host check of the staged copies' threads (ss_shares.h): where the system
gives no more threads, or no memory for one, every share still runs once and
the process goes on (a joinable thread that is destroyed ends it)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def emul(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    out = str(tmp_path_factory.mktemp("shares") / "shares_emul")
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I", os.path.join(ROOT, "poker-solver_b200", "csrc"),
                    os.path.join(ROOT, "tests", "native", "shares_emul.cpp"), "-o", out], check=True)
    return out


@pytest.mark.parametrize("memory", [0, 1])
@pytest.mark.parametrize("shares,threads", [(1, 0), (2, 0), (2, 1), (8, 0), (8, 1), (8, 6), (8, 7)])
def test_every_share_runs_once(emul, shares, threads, memory):
    r = subprocess.run([emul, str(shares), str(threads), str(memory)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    assert [int(x) for x in r.stdout.split()] == [1] * shares + [0] * (8 - shares)
