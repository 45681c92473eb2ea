"""bench.py's reference arm: no port of the reference under its name."""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("workload", [None, "f2-vit", "serve", "calibrate"])
def test_reference_arm_says_unavailable(workload):
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--gpus", "1", "--steps", "2", "--warmup", "3"]
                       + (["--workload", workload] if workload else []),
                       cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout)
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
