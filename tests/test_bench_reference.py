"""bench.py's reference arm where the reference's step code is not built: one line that says so, exit 0."""
import json
import subprocess
import sys
from pathlib import Path

import pytest

from oracle import ref_step

ROOT = Path(__file__).resolve().parents[1]


@pytest.mark.skipif(ref_step.available("step_wgf_f64") and ref_step.available("step_dyn_f64"),
                    reason="the reference's step code is built")
def test_reference_arm_says_unavailable():
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--steps", "1", "--warmup", "3"], cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"]
