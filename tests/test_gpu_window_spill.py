"""Window ranges estimated from every 16th chunk of keys: with a few sampled
chunks per bucket some windows receive more than their range, and the rest is
counted by the global kernel and its low.bin records looked up there."""
import pytest

import kmertreecounter_b200 as kc
import oracle
import torch
from kmertreecounter_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,reads", [(31, 300_000), (63, 400_000)])
def test_spilled_keys(monkeypatch, k, reads):
    monkeypatch.setenv("KC_WINDOW_COUNT", "1")
    data = synth.fastq(synth.params(seed=k, genome_len=5 * reads, n_reads=reads, read_len=(150, 150)))
    keys, counts, K = oracle.count(data, k)
    d = torch.from_numpy(data).cuda()
    with kc.Counter(k=k) as c:
        c.count_device(d.data_ptr(), data.size)
        assert 0 < c.window_spill() < K // 10
        h, distinct = c.histogram(1, 5000)
        assert c.stats.total_kmers == K and distinct == keys.shape[0]
        assert [int(v) for v in h] == [int(v) for v in oracle.histogram(counts, 1, 5000)]
        low, (roots, _) = c.low_bytes(), c.root_records()
        assert low.size // kc.packed_bytes(k) + int(roots["count"].sum(dtype="u8")) == K
