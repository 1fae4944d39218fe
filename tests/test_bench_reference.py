"""The reference arm of bench.py: the reference cannot be built here, and nothing of this
repository stands in for it."""
import json
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_reference_arm_says_unavailable():
    r = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--gpus", "1",
                        "--steps", "3", "--warmup", "3"], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout)
    assert line["impl"] == "reference" and "deal.II" in line["unavailable"] and "value" not in line
