"""bench.py's reference arm without a build of the reference: one JSON line that
says so, and exit code 0. CPU only."""
import json
import os
import subprocess
import sys

import pytest

from oracle_bind import ref_available

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_reference_arm_says_that_it_is_absent():
    if ref_available("fast") or ref_available("strict"):
        pytest.skip("the reference is built here")
    out = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--steps", "1", "--warmup", "1"],
                         cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr[-2000:]
    lines = [ln for ln in out.stdout.splitlines() if ln.startswith("{")]
    assert len(lines) == 1
    d = json.loads(lines[0])
    assert d["impl"] == "reference" and "\n" not in d["unavailable"] and d["unavailable"]
