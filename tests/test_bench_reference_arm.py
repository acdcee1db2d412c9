"""bench.py --impl reference reports the reference or that it is not there: no
figure of this repository's own restatement under the reference's name."""
import json
import os
import subprocess
import sys

from conftest import ROOT


def test_reference_arm_is_unavailable_without_the_reference():
    r = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--steps", "1", "--warmup", "0"],
                       capture_output=True, text=True, timeout=300, cwd=ROOT)
    assert r.returncode == 0, r.stderr[-2000:]
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
