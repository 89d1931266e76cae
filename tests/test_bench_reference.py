"""bench.py --impl reference times the reference solver or says that it cannot: never another solver."""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_reference_arm_without_the_reference():
    if os.path.exists(os.path.join(ROOT, "oracle", "_ref", "spns_ref")):
        pytest.skip("the reference solver is built here")
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--steps", "1", "--warmup", "3", "--ref-sample-n", "32"],
                       cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-500:]
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and set(line) == {"impl", "unavailable"} and "\n" not in line["unavailable"]
