"""`bench.py --impl reference` times the reference or says that it cannot:
without the reference's library it names no other code's time."""
import json
import subprocess
import sys

import pytest

import oracle as O
from conftest import REPO


def test_without_the_reference_the_arm_is_unavailable():
    if O.ref_lib(big=True) is not None:
        pytest.skip("the reference's CPU MPT is built")
    r = subprocess.run([sys.executable, str(REPO / "bench.py"), "--impl", "reference", "--steps", "1", "--warmup", "1"],
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and "unavailable" in line and "value" not in line
