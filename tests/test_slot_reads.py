"""256-bit table slots read while their key arrives, on the host."""
import os
import subprocess

import pytest

from conftest import ROOT
from test_kernel_helpers import NVCC


@pytest.mark.skipif(not os.path.exists(NVCC), reason="nvcc not available")
def test_unfenced_reads(tmp_path):
    exe = tmp_path / "claim_test"
    subprocess.check_call([NVCC, "-std=c++20", "-O2", "-gencode", "arch=compute_100a,code=sm_100a",
                           os.path.join(ROOT, "tests", "native", "claim_test.cu"), "-o", str(exe)])
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.startswith("ok"), out.stdout + out.stderr
