"""bench.py --impl reference: one JSON line that says why the reference cannot
be run, with no number of another program in its place, and exit code 0."""
import json
import os
import subprocess
import sys

from conftest import ROOT


def test_reference_arm_is_unavailable():
    out = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--steps", "1"],
                         capture_output=True, text=True, cwd=ROOT)
    assert out.returncode == 0, out.stderr
    line = json.loads(out.stdout.strip())
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
