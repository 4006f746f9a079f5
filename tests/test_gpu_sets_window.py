"""Read sets counted in windows (a pass of millions of 64-bit keys) against the
oracle and the global count: chunks that span sets, empty and tiny sets between
large ones, buckets of one and of many windows, tables that overflow, and
repeated calls on one context."""
import numpy as np
import pytest

import kmertreecounter_b200 as kc
import oracle
import parity
import torch
from kmertreecounter_b200 import synth

pytestmark = pytest.mark.gpu

KS = (31, 21, 32, 17)


def _sets(reads, genome, seed):
    parts, sets, datas, off = [], [], [], 0
    for i, n in enumerate(reads):
        d = synth.fastq(synth.params(seed=seed + i, genome_len=genome, n_reads=n, read_len=(60 + 7 * i % 90, 150))) \
            if n else np.zeros(0, np.uint8)
        pad = np.full(-d.size % 16, ord("\n"), np.uint8)
        sets.append((off, d.size, KS[i % len(KS)]))
        datas.append(d)
        parts += [d, pad]
        off += d.size + pad.size
    return torch.from_numpy(np.concatenate(parts)).cuda(), sets, datas


@pytest.mark.parametrize("reads,genome,knobs", [
    ([40_000, 0, 3, 60_000, 1, 0, 25_000, 300], 200_000, {}),          # 20x and more, tiny sets between
    ([45_000, 50_000, 20_000], 3_000_000, {}),                          # 2x: tables overflow and grow
    ([400] * 130 + [30_000], 50_000, {}),                               # sets smaller than a chunk
    ([150_000, 7], 3_000_000, {"repeat_ratio": 0.5, "table_load": 0.3}),  # several windows per bucket
])
def test_windowed_sets_match_oracle(monkeypatch, reads, genome, knobs):
    buf, sets, datas = _sets(reads, genome, seed=len(reads))
    want = [oracle.count(d, k) for d, (_, _, k) in zip(datas, sets)]
    assert sum(w[2] for w in want) > 4 << 20  # large enough for windows
    for env in ("1", "0"):
        monkeypatch.setenv("KC_WINDOW_COUNT", env)
        with kc.Counter(k=31, **knobs) as c:
            for _ in range(2):
                res = c.count_sets(buf.data_ptr(), sets)
                low_all, (roots_all, _) = c.low_bytes(), c.root_records()
                for (o, n, k), r, (keys, counts, K) in zip(sets, res, want):
                    low = oracle.unpack(low_all[r.low_offset:r.low_offset + r.low_bytes], k)
                    rec = roots_all[r.root_offset:r.root_offset + r.root_records]
                    parity.check_layout(low, rec, list(r.root_counts), k)
                    mk, mc = parity.merged(low, rec, k)
                    assert r.total_kmers == K
                    assert np.array_equal(mk, keys) and np.array_equal(mc, counts.astype(np.uint64))
            assert c.sets_graph_instantiations() == 1
