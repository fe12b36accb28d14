"""The bench's reference arm runs nothing of this library: where the reference
is not installed it prints one line that says why, and succeeds."""
import json
import os
import subprocess
import sys

from conftest import ROOT


def test_reference_arm_is_unavailable_and_says_why():
    p = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--steps", "3", "--warmup", "3"],
                       capture_output=True, text=True, timeout=120)
    assert p.returncode == 0, p.stderr
    line = json.loads(p.stdout)
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
