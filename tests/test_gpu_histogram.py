"""kc_histogram and kc_bucket_loads against the oracle's exact counts, over
the ways a result can be held: counted in windows (64-bit keys looked up in
staged cells), by the global kernel, in several passes, with grown tables,
and every low.bin record width and key width of the lookup kernels."""
import numpy as np
import pytest

import kmertreecounter_b200 as kc
import oracle
from kmertreecounter_b200 import sizing, synth

pytestmark = pytest.mark.gpu


def _data(scale):
    """Genome-scale reads, then reads of one base and of a short repeat:
    keys with counts far above the shared-memory bins."""
    d = synth.fastq(synth.genome_scale(seed=31, scale=scale))
    hot = b"".join(b"@h%d\n%s\n+\n%s\n" % (i, s, b"I" * 180) for i, s in
                   enumerate([b"A" * 180] * 20 + [b"ACGGT" * 36] * 20))
    return np.concatenate([d, np.frombuffer(hot, np.uint8)])


def _want(keys, counts):
    hi = keys[:, 0]
    model = (hi >> np.uint64(52)).astype(np.int64)
    return (counts.astype(np.int64), np.bincount(model, minlength=4096),
            np.bincount(model, weights=counts.astype(np.float64), minlength=4096).astype(np.int64))


def _check(c, want):
    counts, distinct, kmers = want
    for lo, hi in ((1, 10000), (2, 40), (400, 700), (1, 1)):
        h, d = c.histogram(lo, hi)
        assert d == counts.size
        inside = counts[(counts >= lo) & (counts <= hi)]
        assert np.array_equal(h.astype(np.int64), np.bincount(inside - lo, minlength=hi - lo + 1))
    d, _, km = sizing.bucket_loads(c)
    assert np.array_equal(d.astype(np.int64), distinct) and np.array_equal(km.astype(np.int64), kmers)


@pytest.mark.parametrize("k,buckets", [(31, 256), (31, 4096), (32, 256), (21, 256), (25, 256), (17, 4096), (33, 256),
                                       (47, 4096), (63, 256), (64, 256), (65, 256), (97, 4096), (101, 256), (128, 256)])
def test_histogram_matches_oracle(monkeypatch, k, buckets):
    data = _data(0.004)
    keys, counts, _ = oracle.count(data, k)
    want = _want(keys, counts)
    for env in ("1", "0") if k <= 32 else ("1",):
        monkeypatch.setenv("KC_WINDOW_COUNT", env)
        with kc.Counter(k=k, n_buckets=buckets) as c:
            c.count_host(data)  # one pass
            _check(c, want)
    monkeypatch.delenv("KC_WINDOW_COUNT")
    with kc.Counter(k=k, n_buckets=buckets, batch_bytes=4 << 20) as c:
        assert c.count_host(data).batches > 1
        _check(c, want)
    with kc.Counter(k=k, n_buckets=buckets, bloom_bits=1.0, repeat_ratio=0.002) as c:
        assert c.count_host(data).rehashes > 0 or buckets == 4096
        _check(c, want)


def test_histogram_of_spilled_windows():
    """Window ranges estimated from every 16th chunk, then keys the sample did
    not see: the spilled keys' low.bin records are looked up globally."""
    data = _data(0.04)
    keys, counts, _ = oracle.count(data, 31)
    with kc.Counter(k=31) as c:
        c.count_host(data)
        _check(c, _want(keys, counts))


def test_histogram_of_empty_and_tiny_inputs():
    for data in (b"", b"@r\nACGT\n+\nIIII\n", b"@r\n" + b"ACGTTGCATG" * 5 + b"\n+\n" + b"I" * 50 + b"\n"):
        with kc.Counter(k=31) as c:
            c.count_host(data)
            keys, counts, _ = oracle.count(np.frombuffer(data, np.uint8), 31)
            _check(c, _want(keys, counts))
