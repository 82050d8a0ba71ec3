"""The benchmark's reference arm runs the reference's own library or says that it is
absent; it never times this repository's restatement in its place."""
import json
import os
import subprocess
import sys

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_reference_arm_without_the_reference():
    from oracle import oracle
    if oracle.have_reference():
        pytest.skip("the reference's library is here")
    run = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--steps", "1",
                          "--warmup", "0"], cwd=REPO, capture_output=True, text=True, timeout=600)
    assert run.returncode == 0, run.stderr
    line = json.loads(run.stdout.splitlines()[-1])
    assert line["impl"] == "reference" and "value" not in line
    assert "absent" in line["unavailable"]
