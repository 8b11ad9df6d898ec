"""bench.py --impl reference without the reference's library: it says so and
times nothing in its place."""
import json
import os
import subprocess
import sys

import pytest

from oracle import lib as olib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_reference_arm_without_the_reference(oracles):
    if oracles[0] is not None or os.path.exists(olib.REF_LIB):
        pytest.skip("the reference's library is here")
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--gpus", "1", "--steps", "1", "--warmup",
                        "3"], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert set(line) == {"impl", "unavailable"} and line["impl"] == "reference"
