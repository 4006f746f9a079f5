"""A table that the repeated keys of its bucket fill to the last cell holds them
all: long probe sequences that end at the key itself are no overflow, and no
table grows."""
import numpy as np
import pytest

import kmertreecounter_b200 as kc
import oracle
import parity
import torch
from test_zz_no_alloc import merged_from, noalloc

pytestmark = pytest.mark.gpu

BUCKET = 77


def _reads(k, distinct, copies, seed):
    """`copies` rounds of `distinct` reads of k bases whose canonical keys share their first 8 bits."""
    rng = np.random.default_rng(seed)
    codes = rng.integers(0, 4, (4 * distinct, k), dtype=np.uint8)
    codes[:, :4] = [(BUCKET >> s) & 3 for s in (6, 4, 2, 0)]  # the key's first bases
    codes[:, k - 1] = 0  # the other orientation starts with 3: this one is the smaller
    flip = 3 - codes[:, ::-1]
    assert all(tuple(a) < tuple(b) for a, b in zip(codes, flip))
    codes = np.unique(codes, axis=0)[:distinct]
    seqs = [np.frombuffer(b"ACGT", np.uint8)[3 - row].tobytes() for row in codes]  # complement in read order
    order = [seqs[i] for _ in range(copies) for i in rng.permutation(distinct)]
    return np.frombuffer(b"".join(b"@r\n%s\n+\n%s\n" % (s, b"I" * k) for s in order), np.uint8)


@pytest.mark.parametrize("k,slots", [(31, 512), (63, 256)])
def test_exactly_full_table(monkeypatch, k, slots):
    monkeypatch.setenv("KC_WINDOW_COUNT", "0")
    data = _reads(k, slots, 120, seed=k)
    keys, counts, K = oracle.count(data, k)
    assert keys.shape[0] == slots and set((keys[:, 0] >> np.uint64(56)).tolist()) == {BUCKET}
    with kc.Counter(k=k, repeat_ratio=1e-6, bloom_bits=0.1) as c:
        st = c.count_host(data)
        assert st.max_bucket_table_slots == slots
        parity.check_exact(c, data, k, (keys, counts, K))
        assert st.table_keys == slots and st.rehashes == 0


@pytest.mark.parametrize("k", [31, 63])
def test_exactly_full_table_without_allocation(k):
    data = _reads(k, 64, 100, seed=k)
    keys, counts, _ = oracle.count(data, k)
    cfg = kc.default_config(k=k, repeat_ratio=1e-6, bloom_bits=0.1)
    rc, st, low, roots = noalloc(cfg, torch.from_numpy(data.copy()).cuda(), data.size, 1 << 20, 1 << 20)
    assert rc == 0 and st.rehashes == 0 and st.table_keys == 64
    n = st.low_records * kc.packed_bytes(k)
    (mk, mc), _, _ = merged_from(low.cpu().numpy()[:n], roots.cpu().numpy()[:st.root_records * kc.record_bytes(k)], k,
                                 st.root_records)
    assert np.array_equal(mk, keys) and np.array_equal(mc, counts.astype(np.uint64))


@pytest.mark.parametrize("k,slots", [(31, 512), (63, 256)])
@pytest.mark.parametrize("over", [-40, 1, 60])
def test_nearly_full_and_overfull_tables(monkeypatch, k, slots, over):
    """Keys that end far from their first cell, several occurrences together in a segment's back."""
    monkeypatch.setenv("KC_WINDOW_COUNT", "0")
    data = _reads(k, slots + over, 30, seed=100 + k + over)
    lines = data.tobytes().split(b"\n")[1::4]
    hot = b"".join(b"@h\n%s\n+\n%s\n" % (s, b"I" * k) for s in lines[:slots + over] for _ in range(7))
    data = np.concatenate([data, np.frombuffer(hot, np.uint8), data])
    want = oracle.count(data, k)
    with kc.Counter(k=k, repeat_ratio=1e-6, bloom_bits=0.1) as c:
        for _ in range(2):
            st = c.count_host(data)
            parity.check_exact(c, data, k, want)
            assert (st.rehashes > 0) == (over > 0)
