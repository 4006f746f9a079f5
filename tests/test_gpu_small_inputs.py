"""Small inputs, whose packing and export follow the count without a wait:
sizes from one read up, several passes (only the last one goes ahead), tables
that turn out too small and grow after the export was enqueued, sorted roots,
count filters, repeated calls, and routed keys."""
import numpy as np
import pytest

import kmertreecounter_b200 as kc
import oracle
import parity
import torch
from kmertreecounter_b200 import synth

pytestmark = pytest.mark.gpu


def _reads(n, seed=5, genome=40_000):
    return synth.fastq(synth.params(seed=seed, genome_len=genome, n_reads=n, read_len=(120, 150)))


@pytest.mark.parametrize("k", [21, 31, 47, 101])
def test_sizes_from_one_read(k):
    with kc.Counter(k=k) as c:
        for n in (1, 2, 50, 1000, 9000, 3):  # one context: buffers of a larger call serve a smaller one
            data = _reads(n, seed=n)
            d = torch.from_numpy(data).cuda()
            for _ in range(2):
                c.count_device(d.data_ptr(), d.numel())
                parity.check_exact(c, data, k)
            keys, counts, _ = oracle.count(data, k)
            h, distinct = c.histogram(1, 300)
            assert distinct == keys.shape[0]
            assert [int(x) for x in h] == [int(x) for x in oracle.histogram(counts, 1, 300)]


@pytest.mark.parametrize("k", [31, 63, 101])
@pytest.mark.parametrize("buckets", [256, 4096])
def test_growth_after_the_export_was_enqueued(k, buckets):
    data = _reads(20_000, genome=300_000)
    with kc.Counter(k=k, n_buckets=buckets, repeat_ratio=1e-6, bloom_bits=0.1) as c:
        for _ in range(2):
            st = c.count_host(data)
            assert st.rehashes > 0 or buckets == 4096  # 4096 tables of the smallest size hold these keys
            parity.check_exact(c, data, k)
    with kc.Counter(k=k, n_buckets=buckets, repeat_ratio=1e-6, bloom_bits=0.1, batch_bytes=1 << 20,
                    sort_output=1) as c:
        st = c.count_host(data)
        assert (st.rehashes > 0 or buckets == 4096) and st.batches > 1
        _, roots = parity.check_exact(c, data, k)
        w = roots["key"].reshape(roots.shape[0], -1)
        order = np.lexsort([w[:, i] for i in range(w.shape[1] - 1, -1, -1)])
        assert np.array_equal(order, np.arange(w.shape[0]))


def test_filter_and_routed_keys():
    data = _reads(4000)
    with kc.Counter(k=31, min_count=2, max_count=9) as c:
        c.count_host(data)
        parity.check_filtered(c, data, 31, 2, 9)
    d = torch.from_numpy(data).cuda()
    with kc.Counter(k=31) as c:
        counts = c.route_device(d.data_ptr(), d.numel())
        addr, n = c.routed_keys()
        keys = torch.empty(n, dtype=torch.int64, device="cuda")
        c.copy_routed(keys.data_ptr(), 8 * n)
        c.count_keys_device(keys.data_ptr(), n, counts)
        parity.check_exact(c, data, 31)
