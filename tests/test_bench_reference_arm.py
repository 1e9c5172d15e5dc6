"""The bench's reference arm where the reference is not built: one line that
says so, and success."""

import json
import os
import subprocess
import sys

import pytest

from oracle import refmpi

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(os.path.exists(refmpi.MPI_LIB), reason="the reference is built here")
def test_unavailable_line():
    out = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--steps", "2", "--warmup", "3"], cwd=ROOT,
                         capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    line = json.loads(out.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"]
