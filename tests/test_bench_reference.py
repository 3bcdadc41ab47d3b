"""bench.py --impl reference times the reference's own library or says that it is
unavailable; it never stands in for it."""
import json
import os
import subprocess
import sys

import pytest

from oracle import refbridge

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(refbridge.available(), reason="the reference's library is built here")
def test_reference_arm_without_the_reference():
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--steps", "1", "--warmup", "0"], cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
