"""Host check of the value/regret kernel's 32-bit numbering of (item, pair of
hands) units: a level with more of them than 2^31, which a batch of many small
subgames beside one of 1326 hands can have, is cut into launches."""
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
    out = str(tmp_path_factory.mktemp("cfv") / "cfv_units")
    inc = [os.path.join(ROOT, "include"), os.path.join(ROOT, "poker-solver_b200", "csrc")]
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", inc[0], "-I", inc[1],
                    os.path.join(ROOT, "tests", "native", "cfv_units.cpp"), "-o", out], check=True)
    return out


@pytest.mark.parametrize("items,hands,launches", [
    (1, 1, 1), (1, 1326, 1), (21436, 1128, 1), (3376 * 1130, 1128, 2), (3239040, 1326, 1), (3239041, 1326, 2),
    (2147483520, 2, 1), (2147483647, 2, 2), (2147483647, 3, 3), (2147483647, 1326, 664),
])
def test_units_stay_in_32_bits(emul, items, hands, launches):
    res = json.loads(subprocess.run([emul, str(items), str(hands)], capture_output=True, text=True, check=True).stdout)
    assert res == {"launches": launches, "covered": items, "good": 1}
