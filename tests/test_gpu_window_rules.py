"""Which counts take shared-memory windows (the sub-routing stage runs), by size
and with KC_WINDOW_COUNT=0/1, and that both forms agree with the oracle where
buckets have many windows: default sizing knobs, whose tables have fewer than
half a cell per key."""
import numpy as np
import pytest

import kmertreecounter_b200 as kc
import oracle
import parity
import torch
from kmertreecounter_b200 import synth

pytestmark = pytest.mark.gpu


def _reads(n, genome=200_000, length=150, seed=11):
    return synth.fastq(synth.params(seed=seed, genome_len=genome, n_reads=n, read_len=(length, length)))


def _windowed(c):
    return c.stage_times()["subroute"][1] > 0


@pytest.mark.parametrize("k,reads,by_size", [(31, 3_000, True), (63, 20_000, False), (47, 100_000, False),
                                             (63, 600_000, True), (64, 600_000, False)])
def test_one_input(monkeypatch, k, reads, by_size):
    data = _reads(reads)
    d = torch.from_numpy(data).cuda()
    spectra = []
    for env, want in ((None, by_size), ("0", False), ("1", k <= 63)):
        monkeypatch.delenv("KC_WINDOW_COUNT", raising=False)
        if env:
            monkeypatch.setenv("KC_WINDOW_COUNT", env)
        with kc.Counter(k=k) as c:
            c.count_device(d.data_ptr(), data.size)
            assert _windowed(c) == want, env
            h, distinct = c.histogram(1, 5000)
            spectra.append((int(c.stats.total_kmers), distinct, [int(v) for v in h]))
    assert spectra[1:] == spectra[:-1]


@pytest.mark.parametrize("k,reads,buckets", [(31, 60_000, 256), (21, 60_000, 256), (63, 60_000, 256), (47, 60_000, 256)])
def test_many_windows_per_bucket(monkeypatch, k, reads, buckets):
    data = _reads(reads)
    d = torch.from_numpy(data).cuda()
    want = oracle.count(data, k)
    for env in ("1", "0"):
        monkeypatch.setenv("KC_WINDOW_COUNT", env)
        with kc.Counter(k=k, n_buckets=buckets) as c:
            st = c.count_device(d.data_ptr(), data.size)
            assert _windowed(c) == (env == "1")
            assert st.max_bucket_table_slots > (4096 if k <= 32 else 2048)  # the cells of one window
            parity.check_exact(c, data, k, want)


@pytest.mark.parametrize("sets,reads,by_size", [(400, 400, False), (6, 60_000, True)])
def test_read_sets(monkeypatch, sets, reads, by_size):
    """A pass of many small sets has few keys for each window."""
    one = _reads(reads, genome=max(2000, reads))
    pad = np.full(-one.size % 16, ord("\n"), np.uint8)
    part = torch.from_numpy(np.concatenate([one, pad])).cuda()
    buf = part.repeat(sets)
    desc = [(i * part.numel(), one.size, 31) for i in range(sets)]
    keys, counts, K = oracle.count(one, 31)
    assert K * sets > 4 << 20
    for env, want in ((None, by_size), ("0", False)):
        monkeypatch.delenv("KC_WINDOW_COUNT", raising=False)
        if env:
            monkeypatch.setenv("KC_WINDOW_COUNT", env)
        with kc.Counter(k=31) as c:
            res = c.count_sets(buf.data_ptr(), desc)
            assert _windowed(c) == want, env
            low_all, (roots_all, _) = c.low_bytes(), c.root_records()
            for r in (res[0], res[sets // 2], res[-1]):
                low = oracle.unpack(low_all[r.low_offset:r.low_offset + r.low_bytes], 31)
                mk, mc = parity.merged(low, roots_all[r.root_offset:r.root_offset + r.root_records], 31)
                assert r.total_kmers == K and np.array_equal(mk, keys) and np.array_equal(mc, counts.astype(np.uint64))
