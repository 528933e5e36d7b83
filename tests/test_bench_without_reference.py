"""bench.py on a machine without the reference's sources: its reference arm says
so in one line and succeeds."""
import json
import os
import subprocess
import sys

import pytest

from oracle.oracle import Reference

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(Reference.available(), reason="the reference is built here")
def test_reference_arm_says_that_it_is_unavailable():
    r = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--steps", "1",
                        "--warmup", "3"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    lines = [json.loads(x) for x in r.stdout.splitlines() if x.startswith("{")]
    assert len(lines) == 1 and lines[0]["impl"] == "reference" and "not built" in lines[0]["unavailable"]
