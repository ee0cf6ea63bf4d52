"""`bench.py --impl reference` runs the reference's own code or says that it is not
there; the repository's restatement never stands in for it."""
import json
import subprocess
import sys
from pathlib import Path

import pytest

import oracle

ROOT = Path(__file__).resolve().parent.parent


def test_without_the_reference_the_arm_says_so():
    if oracle.reference_lib() is not None:
        pytest.skip("the reference's kernel is built here")
    r = subprocess.run([sys.executable, str(ROOT / "bench.py"), "--impl", "reference", "--steps", "1", "--warmup", "0"],
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"]
    assert "value" not in line
