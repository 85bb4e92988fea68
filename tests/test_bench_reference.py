"""`bench.py --impl reference` times the reference's own kernels or says that it
cannot: never this repository's restatement under the reference's name."""

import json
import os
import subprocess
import sys

import pytest

from oracle import pyoracle as O

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(O.reference_available(3, 3), reason="the reference's kernels are built here")
def test_reference_arm_without_the_reference_is_unavailable():
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--steps", "1", "--warmup", "0"],
                       cwd=ROOT, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
