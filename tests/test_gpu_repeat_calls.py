"""The second call on a context finds every buffer of the first: no device
memory is allocated or given back by repeating a count, whatever path it takes."""
import numpy as np
import pytest

import kmertreecounter_b200 as kc
import oracle
import torch
from kmertreecounter_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,k", [("input", 31), ("input", 63), ("input", 101), ("sets", 31), ("routed", 63)])
def test_second_call_allocates_nothing(monkeypatch, form, k):
    monkeypatch.setenv("KC_WINDOW_COUNT", "1")  # windows wherever the key width has them
    data = synth.fastq(synth.params(seed=k, genome_len=1_500_000, n_reads=400_000, read_len=(150, 150)))
    pad = np.full(-data.size % 16, ord("\n"), np.uint8)
    d = torch.from_numpy(np.concatenate([data, pad])).cuda()
    kmers = 400_000 * (150 - k + 1)
    with kc.Counter(k=k) as c:
        torch.cuda.synchronize()
        if form == "routed":
            with kc.Counter(k=k) as r:
                counts = r.route_device(d.data_ptr(), data.size)
                _, n = r.routed_keys()
                keys = torch.empty(2 * n, dtype=torch.int64, device="cuda")
                r.copy_routed(keys.data_ptr(), 16 * n)
        free, got = [], []
        for _ in range(4):
            if form == "sets":
                res = c.count_sets(d.data_ptr(), [(0, data.size, k), (0, data.size // 3, k)])
                got.append((res[0].total_kmers, res[1].total_kmers))
            else:
                if form == "input":
                    c.count_device(d.data_ptr(), data.size)
                else:
                    c.count_keys_device(keys.data_ptr(), n, counts)
                h, distinct = c.histogram(1, 500)
                got.append((int(c.stats.total_kmers), distinct, [int(v) for v in h]))
            free.append(torch.cuda.mem_get_info()[0])
        assert got[1:] == got[:-1] and 0 < got[0][0] <= kmers
        assert free[1:] == free[:-1], [a - free[0] for a in free]


def test_counts_after_the_buffers_changed_places():
    """Windowed, global, routed and multi-pass counts in turn on one context."""
    data = synth.fastq(synth.params(seed=3, genome_len=300_000, n_reads=60_000, read_len=(100, 150)))
    d = torch.from_numpy(data).cuda()
    want = oracle.count(data, 31)
    h_want = [int(v) for v in oracle.histogram(want[1], 1, 300)]

    def check(c):
        h, distinct = c.histogram(1, 300)
        assert c.stats.total_kmers == want[2] and distinct == want[0].shape[0] and [int(v) for v in h] == h_want

    with kc.Counter(k=31, batch_bytes=4 << 20) as c:
        for _ in range(2):
            c.count_device(d.data_ptr(), data.size)
            check(c)
            counts = c.route_device(d.data_ptr(), data.size)
            addr, n = c.routed_keys()
            c.count_keys_device(addr, n, counts)  # the context's own routed keys
            check(c)
            c.count_host(data)
            check(c)
            c.count_sets(d.data_ptr(), [(0, data.size, 31)])
