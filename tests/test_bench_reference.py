"""`bench.py --impl reference` without the reference's binary says so in its one
line, at once, instead of timing something else."""
import json
import os
import subprocess
import sys

import pytest

import oracle
from conftest import ROOT


@pytest.mark.skipif(os.path.exists(oracle.REF_TREE), reason="the reference is built here")
def test_unavailable_line():
    out = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--steps", "1",
                          "--warmup", "0"], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stderr
    line = json.loads(out.stdout.strip())
    assert line["impl"] == "reference" and line["unavailable"]
