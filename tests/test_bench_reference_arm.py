"""`bench.py --impl reference` without the reference program: one JSON line
that says so, no number of this repository's own code in its place."""
import json
import os
import subprocess
import sys

import pytest

from oracle import ref_runner

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(ref_runner.available(omp=True), reason="the reference program is built")
def test_unavailable_line():
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--steps", "1", "--warmup", "1"], cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert set(line) == {"impl", "unavailable"} and line["impl"] == "reference"
