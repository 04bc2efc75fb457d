"""`bench.py --impl reference` times the reference's own CPU pipeline or nothing:
where that is not built, one line says so, and no part of this build runs in its
place."""
import json
import os
import subprocess
import sys

import pytest

import oracle
from conftest import ROOT


def test_reference_arm_says_when_there_is_no_reference():
    if oracle.bullet_lib() is not None:
        pytest.skip("the reference's CPU pipeline is built here")
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--gpus", "1", "--steps", "2", "--warmup", "3"],
                       cwd=ROOT, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
