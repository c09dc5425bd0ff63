"""bench.py --impl reference without the reference's library: one line that says so, and nothing timed."""
import json
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_reference_arm_without_the_library():
    from oracle.oracle import REF_SO
    if REF_SO.exists():
        pytest.skip("the reference library is built")
    res = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--gpus", "1", "--steps", "2", "--warmup", "1"],
                         cwd=ROOT, capture_output=True, text=True, timeout=120)
    assert res.returncode == 0, res.stderr
    line = json.loads(res.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and REF_SO.name in line["unavailable"] and "value" not in line
