"""The sort stage of a sorted count: the launches it reports are those it makes
(five for each digit pass, three for the runs of equal leading bits)."""
import numpy as np
import pytest

import kmertreecounter_b200 as kc
import oracle
import parity
from kmertreecounter_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,genome,reads,want", [
    (31, 150_000, 12_000, 5 * 4 + 3),   # 2^17 records: 26 leading bits, 4 digits of 8
    (63, 150_000, 12_000, 5 * 4 + 3),   # 4 of 16
    (31, 5_000, 400, 5 * 8),            # few records: every digit
    (17, 150_000, 12_000, 5 * 4 + 3),   # 4 of 5
])
def test_reported_launches(k, genome, reads, want):
    data = synth.fastq(synth.params(seed=k, genome_len=genome, n_reads=reads, read_len=(150, 200)))
    with kc.Counter(k=k, sort_output=1) as c:
        c.count_host(data)
        _, roots = parity.check_exact(c, data, k)
        assert (roots.shape[0] >= 1 << 16) == (reads > 400) and roots.shape[0] < 1 << 18
        assert c.stage_times()["sort"][1] == want


@pytest.mark.parametrize("k,length", [(31, 100), (63, 130), (101, 180)])
@pytest.mark.parametrize("tails,heads", [((b"A",), 3000), ((b"A", b"CA", b"CCA"), 1800), ((b"A",), 40_000)])
def test_long_runs(k, length, tails, heads):
    """Reads that end in a repeat put many distinct keys behind one prefix:
    one long run, several (sorted apart), and a run of most of the records."""
    rng = np.random.default_rng(k + heads)
    acgt = np.frombuffer(b"ACGT", np.uint8)
    out = []
    for t in tails:
        tail = np.frombuffer((t * 40)[:40], np.uint8)
        for h in acgt[rng.integers(0, 4, (heads, length - 40))]:
            s = np.concatenate([h, tail]).tobytes()
            out += [b"@p\n%s\n+\n%s\n" % (s, b"I" * length)] * 2
    base = synth.fastq(synth.params(seed=k, genome_len=600_000, n_reads=50_000, read_len=(150, 200)))
    data = np.concatenate([base, np.frombuffer(b"".join(out), np.uint8)])
    want = oracle.count(data, k)
    with kc.Counter(k=k, sort_output=1) as c:
        c.count_host(data)
        _, roots = parity.check_exact(c, data, k, want)
        assert roots.shape[0] > 1 << 18
        w = roots["key"].reshape(roots.shape[0], -1)
        order = np.lexsort([w[:, i] for i in range(w.shape[1] - 1, -1, -1)])
        assert np.array_equal(order, np.arange(w.shape[0]))
        digits = (2 * k + 7) // 8
        assert c.stage_times()["sort"][1] == 5 * 4 + 3 + 5 * digits  # the leading digits, the runs, the long ones
