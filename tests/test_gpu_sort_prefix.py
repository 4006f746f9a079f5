"""Sorted root records when the sort goes over the leading key bits only:
records that agree in all of those (keys behind a common prefix) in runs of a
few, of hundreds, and of more than a block sorts, which takes the passes over
every digit."""
import numpy as np
import pytest

import kmertreecounter_b200 as kc
import oracle
import parity
from kmertreecounter_b200 import synth

pytestmark = pytest.mark.gpu


def _prefix_reads(heads, length, seed):
    """Reads, each twice, of a random head and a tail of 40 A's: the windows
    that end deep in the tail have keys whose leading bases are all A (the
    reverse-order orientation starts with the newest base)."""
    rng = np.random.default_rng(seed)
    acgt = np.frombuffer(b"ACGT", np.uint8)
    out = []
    for i in range(heads):
        s = np.concatenate([acgt[rng.integers(0, 4, length - 40)], np.full(40, ord("A"), np.uint8)]).tobytes()
        out += [b"@p%d\n%s\n+\n%s\n" % (i, s, b"I" * length)] * 2
    return np.frombuffer(b"".join(out), np.uint8)


@pytest.mark.parametrize("k,length", [(31, 100), (47, 110), (101, 180)])
@pytest.mark.parametrize("heads", [3, 90, 4000])
def test_runs_behind_a_common_prefix(k, length, heads):
    base = synth.fastq(synth.params(seed=k, genome_len=150_000, n_reads=12_000, read_len=(150, 200)))
    data = np.concatenate([base, _prefix_reads(heads, length, seed=heads)])
    want = oracle.count(data, k)
    with kc.Counter(k=k, sort_output=1) as c:
        c.count_host(data)
        _, roots = parity.check_exact(c, data, k, want)
        assert roots.shape[0] > 1 << 16  # the leading-bits form's range
        w = roots["key"].reshape(roots.shape[0], -1)
        order = np.lexsort([w[:, i] for i in range(w.shape[1] - 1, -1, -1)])
        assert np.array_equal(order, np.arange(w.shape[0]))
