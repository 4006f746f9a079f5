"""Compile the stream form of the k-mer keys (kc_kernels.cuh) for the host and
check it, the sequence-line mask and the run mask against their definitions
(CPU only)."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.mark.skipif(not os.path.exists(NVCC), reason="nvcc not available")
def test_stream_keys(tmp_path):
    exe = tmp_path / "streams_test"
    subprocess.check_call([NVCC, "-std=c++20", "-O2", "-gencode", "arch=compute_100a,code=sm_100a",
                           os.path.join(ROOT, "tests", "native", "streams_test.cu"), "-o", str(exe)])
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr
    assert out.stdout.startswith("streams ok")
