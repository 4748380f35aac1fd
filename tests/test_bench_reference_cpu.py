"""bench.py's reference arm: without a build of the reference's own sources it
says so, and measures nothing in their place."""
import json
import os
import subprocess
import sys

import pytest

from oracle import oracle

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(oracle.ref_available(), reason="the reference is built")
def test_reference_arm_without_reference():
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--gpus", "1", "--steps", "3", "--warmup", "3"],
                       cwd=ROOT, env=dict(os.environ, NS3D_REF_DIR=os.path.join(ROOT, "tests")), capture_output=True, text=True)
    assert r.returncode == 0
    line = json.loads(r.stdout.splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
