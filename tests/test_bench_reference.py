"""bench.py's reference arm without the reference: one line that says so, and success."""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(os.path.exists(os.path.join(ROOT, "oracle", "_ref", "libanalogsat_ref.so")),
                    reason="the reference is built here")
def test_reference_arm_says_that_it_is_unavailable():
    r = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--gpus", "1",
                        "--steps", "2", "--warmup", "1"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    lines = r.stdout.strip().splitlines()
    assert len(lines) == 1
    line = json.loads(lines[0])
    assert line["impl"] == "reference" and "\n" not in line["unavailable"] and line["unavailable"]
