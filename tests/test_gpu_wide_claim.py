"""256-bit keys: slots claimed half by half (k <= 127) and by the published
state (k = 128) against the oracle: keys that share their first half, halves
with words of all ones, hot keys, tables that overflow and grow, several
passes, and read sets with and without a k of 128."""
import numpy as np
import pytest

import kmertreecounter_b200 as kc
import oracle
import parity
import torch
from kmertreecounter_b200 import synth

pytestmark = pytest.mark.gpu


def _data():
    rng = np.random.default_rng(7)
    acgt = np.frombuffer(b"ACGT", np.uint8)
    base = synth.fastq(synth.params(seed=51, genome_len=60_000, n_reads=12_000, read_len=(140, 200)))
    recs = []
    for stem in range(4):  # windows that share their leading 64 bases, in either orientation
        head = acgt[rng.integers(0, 4, 100)]
        for _ in range(2):
            tails = np.random.default_rng(stem)
            for i in range(300):
                t = acgt[tails.integers(0, 4, 70)]
                recs.append((np.concatenate([head, t]) if stem % 2 else np.concatenate([t, head])).tobytes())
    for s in (b"A" * 170, b"T" * 170, b"A" * 63 + b"T" * 107, b"A" * 80 + b"T" * 90, b"CA" + b"T" * 64 + b"AC" * 40):
        recs += [s] * 200
    text = b"".join(b"@r\n%s\n+\n%s\n" % (s, b"I" * len(s)) for s in recs)
    return np.concatenate([base, np.frombuffer(text, np.uint8)])


@pytest.mark.parametrize("k", [65, 95, 101, 127, 128])
def test_wide_claims(k):
    data = _data()
    d = torch.from_numpy(data).cuda()
    want = oracle.count(data, k)
    for knobs in ({}, dict(bloom_bits=1.0, repeat_ratio=0.002), dict(n_buckets=4096),
                  dict(device_batch_bytes=data.size // 3 // 8192 * 8192)):
        with kc.Counter(k=k, **knobs) as c:
            c.count_device(d.data_ptr(), d.numel())
            parity.check_exact(c, data, k, want)
            h, distinct = c.histogram(1, 4000)
            assert distinct == want[0].shape[0]
            assert [int(v) for v in h] == [int(v) for v in oracle.histogram(want[1], 1, 4000)]


@pytest.mark.parametrize("ks", [(101, 127, 65), (128, 101, 127)])
def test_wide_sets(ks):
    datas = [_data(), _data()[:200_000 // 8 * 8], _data()]
    datas[1] = datas[1][:int(np.flatnonzero(datas[1] == ord("\n"))[-1]) + 1]
    sets, parts, off = [], [], 0
    for x, k in zip(datas, ks):
        pad = np.full(-x.size % 16, ord("\n"), np.uint8)
        sets.append((off, x.size, k))
        parts += [x, pad]
        off += x.size + pad.size
    buf = torch.from_numpy(np.concatenate(parts)).cuda()
    for knobs in ({}, dict(repeat_ratio=0.002)):
        with kc.Counter(k=101, **knobs) as c:
            res = c.count_sets(buf.data_ptr(), sets)
            low_all, (roots_all, _) = c.low_bytes(), c.root_records()
            for x, (o, n, k), r in zip(datas, sets, res):
                keys, counts, K = oracle.count(x, k)
                low = oracle.unpack(low_all[r.low_offset:r.low_offset + r.low_bytes], k)
                rec = roots_all[r.root_offset:r.root_offset + r.root_records]
                mk, mc = parity.merged(low, rec, k)
                assert r.total_kmers == K
                assert np.array_equal(mk, keys) and np.array_equal(mc, counts.astype(np.uint64))
