"""128-bit keys counted in shared-memory windows (one device pass, k <= 63)
against the oracle and the global count: keys that share their first word (the
two-step claim of a cell), hot keys, buckets of one and of many windows, tables
that overflow and grow, later passes on the same tables, the merged histogram,
and routed keys."""
import numpy as np
import pytest

import kmertreecounter_b200 as kc
import oracle
import parity
import torch
from kmertreecounter_b200 import synth

pytestmark = pytest.mark.gpu


def _data(scale=0.004):
    rng = np.random.default_rng(3)
    acgt = np.frombuffer(b"ACGT", np.uint8)
    base = synth.fastq(synth.genome_scale(seed=41, scale=scale))
    recs = []
    for stem in range(4):  # windows that end in a tail share their oldest bases, in either orientation
        head = acgt[rng.integers(0, 4, 70)]
        tails = [acgt[rng.integers(0, 4, 50)] for _ in range(400)]
        for i, t in enumerate(tails * 2):
            s = (np.concatenate([head, t]) if stem % 2 else np.concatenate([t, head])).tobytes()
            recs.append(b"@s%d\n%s\n+\n%s\n" % (i, s, b"I" * len(s)))
    recs += [b"@h\n%s\n+\n%s\n" % (b"A" * 160, b"I" * 160)] * 300
    return np.concatenate([base, np.frombuffer(b"".join(recs), np.uint8)])


@pytest.mark.parametrize("k", [33, 47, 63, 64])
@pytest.mark.parametrize("buckets", [256, 4096])
def test_windowed_long_keys(monkeypatch, k, buckets):
    data = _data()
    d = torch.from_numpy(data).cuda()
    keys, counts, K = oracle.count(data, k)
    for env in ("1", "0"):
        monkeypatch.setenv("KC_WINDOW_COUNT", env)
        for knobs in ({}, dict(bloom_bits=1.0, repeat_ratio=0.002), dict(repeat_ratio=0.3, table_load=0.5)):
            with kc.Counter(k=k, n_buckets=buckets, **knobs) as c:
                st = c.count_device(d.data_ptr(), d.numel())
                assert st.batches == 1
                parity.check_exact(c, data, k, (keys, counts, K))
                h, distinct = c.histogram(1, 2000)
                assert distinct == keys.shape[0]
                assert [int(v) for v in h] == [int(v) for v in oracle.histogram(counts, 1, 2000)]


def test_later_passes_and_routed_keys():
    data = _data(0.02)
    d = torch.from_numpy(data).cuda()
    want = oracle.count(data, 55)
    # passes of a third: the first may be counted in windows, the last is small
    with kc.Counter(k=55, device_batch_bytes=data.size // 3 // 8192 * 8192) as c:
        assert c.count_device(d.data_ptr(), d.numel()).batches > 2
        parity.check_exact(c, data, 55, want)
    with kc.Counter(k=55) as c:
        counts = c.route_device(d.data_ptr(), d.numel())
        _, n = c.routed_keys()
        keys = torch.empty(2 * n, dtype=torch.int64, device="cuda")
        c.copy_routed(keys.data_ptr(), 16 * n)
        c.count_keys_device(keys.data_ptr(), n, counts)
        parity.check_exact(c, data, 55, want)
