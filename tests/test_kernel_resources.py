"""Kernels whose speed rests on keeping their state in registers: no spills in
ptxas's report (compiled here, no GPU)."""
import os
import re
import subprocess

import pytest

from conftest import ROOT
from test_kernel_helpers import NVCC


@pytest.mark.skipif(not os.path.exists(NVCC), reason="nvcc not available")
def test_count_keeps_its_registers(tmp_path):
    out = subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++20",
                          "--expt-relaxed-constexpr", "-Xptxas", "-v", "-cubin",
                          os.path.join(ROOT, "tests", "native", "resources.cu"), "-o", str(tmp_path / "r.cubin")],
                         capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stderr
    spills = re.findall(r"Compiling entry function '(\S*count_routed\S*)'.*?(\d+) bytes spill stores, (\d+) bytes spill loads",
                        out.stderr, re.S)
    assert len(spills) == 3, out.stderr
    assert all(int(st) == 0 and int(ld) == 0 for _, st, ld in spills), spills
