"""The sort stage of a sorted count: the launches it reports are those it makes
(five for each digit pass, three for the runs of equal leading bits)."""
import pytest

import kmertreecounter_b200 as kc
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
