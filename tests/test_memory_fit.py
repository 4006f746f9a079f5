"""Key buffers against the device's memory: the rule on the host, and a
multi-set pass on a device that has room for one key buffer but not for two."""
import os
import subprocess

import numpy as np
import pytest

import kmertreecounter_b200 as kc
import oracle
import parity
from conftest import ROOT
from kmertreecounter_b200 import synth


def test_rule(tmp_path):
    exe = tmp_path / "fit_test"
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.check_call(["g++", "-std=c++20", "-O1", "-I", os.path.join(cuda, "include"),
                           os.path.join(ROOT, "tests", "native", "fit_test.cpp"), "-o", str(exe)])
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.startswith("ok"), out.stdout + out.stderr


def _counted(c, buf, sets):
    """Per set: k-mers, and k-mers in the outputs; the first set's exact counts."""
    res = c.count_sets(buf.data_ptr(), sets)
    low, (roots, _) = c.low_bytes(), c.root_records()
    part = [roots[r.root_offset:r.root_offset + r.root_records] for r in res]
    totals = [(r.total_kmers, r.low_records + int(q["count"].sum(dtype=np.uint64))) for r, q in zip(res, part)]
    keys, counts = parity.merged(oracle.unpack(low[res[0].low_offset:res[0].low_offset + res[0].low_bytes], 31), part[0], 31)
    return totals, keys, counts


@pytest.mark.gpu
def test_sets_with_room_for_one_key_buffer(monkeypatch):
    import torch
    one = synth.fastq(synth.params(seed=9, genome_len=4_000_000, n_reads=400_000, read_len=(150, 150)))
    pad = np.full(-one.size % 16, ord("\n"), np.uint8)
    part = torch.from_numpy(np.concatenate([one, pad])).cuda()
    buf = part.repeat(3)  # 144 M k-mers: 1.15 GB a key buffer
    sets = [(i * part.numel(), one.size, 31) for i in range(3)]
    torch.cuda.synchronize()

    def held(c):
        free = torch.cuda.mem_get_info()[0]
        got = _counted(c, buf, sets)
        return free - torch.cuda.mem_get_info()[0], got

    # what the pass takes without windows, and what it finds
    monkeypatch.setenv("KC_WINDOW_COUNT", "0")
    with kc.Counter(k=31) as c:
        need, want = held(c)
    monkeypatch.setenv("KC_WINDOW_COUNT", "1")
    c = kc.Counter(k=31)
    room = need + (128 << 20)
    keep = torch.empty(torch.cuda.mem_get_info()[0] - room, dtype=torch.uint8, device="cuda")
    try:
        for _ in range(2):
            got = _counted(c, buf, sets)
            assert got[0] == want[0] and all(a == b for a, b in got[0])
            assert np.array_equal(got[1], want[1]) and np.array_equal(got[2], want[2])
    finally:
        c.close()
        del keep
        torch.cuda.empty_cache()
