"""bench.py --impl reference without the reference's engine (host)."""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))


def test_reference_arm_without_the_engine_is_unavailable():
    """The CPU restatement is not timed in the reference's name."""
    sys.path.insert(0, ROOT)
    from oracle import refio
    if refio.ref_available():
        pytest.skip("the reference's engine is built here")
    r = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--steps", "1",
                        "--warmup", "0"], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
