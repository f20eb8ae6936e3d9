"""bench.py --impl reference: no restatement of the reference's algorithm is
printed under its name."""
import json
import os
import subprocess
import sys

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_reference_arm_says_why_it_cannot_run():
    r = subprocess.run([sys.executable, os.path.join(REPO, "bench.py"), "--impl", "reference", "--gpus", "1", "--steps", "1",
                        "--warmup", "3"], capture_output=True, text=True, timeout=120, cwd=REPO)
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout)
    assert set(line) == {"impl", "unavailable"} and line["impl"] == "reference"
    assert line["unavailable"] and "\n" not in line["unavailable"]
