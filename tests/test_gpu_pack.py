"""low.bin packing for record widths from 1 byte to 4 words: records of every
remainder against 16-byte stores, runs that start and end anywhere in one,
single inputs, read sets with two record widths in one pass, and the
allocation-free entry point (whose output buffer has no slack)."""
import ctypes as C

import numpy as np
import pytest

import kmertreecounter_b200 as kc
import oracle
import parity
import torch
from kmertreecounter_b200 import synth
from kmertreecounter_b200._native import KcStats, check, lib

pytestmark = pytest.mark.gpu


def _reads(n, length, seed):
    return synth.fastq(synth.params(seed=seed, genome_len=60_000, n_reads=n, read_len=(length, length)))


@pytest.mark.parametrize("k", [1, 4, 6, 9, 13, 17, 20, 24, 28, 32, 33, 36, 40, 44, 48, 52, 56, 60, 65, 69, 73, 77, 81,
                               85, 89, 93, 99, 101, 104, 108, 112, 116, 120, 124])
def test_record_widths(k):
    data = _reads(700, 180, k)
    want = oracle.count(data, k)
    with kc.Counter(k=k) as c:
        c.count_host(data)
        parity.check_exact(c, data, k, want)
    with kc.Counter(k=k, batch_bytes=1 << 20, device_batch_bytes=1 << 20) as c:
        big = np.concatenate([data] * 8)  # later passes start mid-vector
        d = torch.from_numpy(big).cuda()
        assert c.count_device(d.data_ptr(), d.numel()).batches > 1
        parity.check_exact(c, big, k)
    if k <= 64:
        cfg = kc.default_config(k=k)
        d = torch.from_numpy(data).cuda()
        low_n = int(want[0].shape[0]) * kc.packed_bytes(k)
        low = torch.full((low_n + 64,), 0xA5, dtype=torch.uint8, device="cuda")
        roots = torch.empty(int(want[2]) * kc.record_bytes(k) + 64, dtype=torch.uint8, device="cuda")
        st = KcStats()
        check(lib.kc_count_device_noalloc(C.byref(cfg), C.c_void_p(d.data_ptr()), d.numel(), C.c_void_p(low.data_ptr()),
                                          low_n, C.c_void_p(roots.data_ptr()), roots.numel(), None, C.byref(st)))
        torch.cuda.synchronize()
        out = low.cpu().numpy()
        used = st.low_records * kc.packed_bytes(k)
        assert np.all(out[used:] == 0xA5)  # nothing past the last record
        keys = oracle.unpack(out[:used], k)
        assert parity.unique_rows(keys) and keys.shape[0] == st.low_records


@pytest.mark.parametrize("ks", [(21, 31, 9, 29), (33, 63, 48, 64), (65, 101, 128, 97)])
def test_sets_of_two_widths(ks):
    parts, sets, datas, off = [], [], [], 0
    for i in range(24):
        d = _reads(1 + 37 * i, 150, 100 + i)
        pad = np.full(-d.size % 16, ord("\n"), np.uint8)
        sets.append((off, d.size, ks[i % len(ks)]))
        datas.append(d)
        parts += [d, pad]
        off += d.size + pad.size
    buf = torch.from_numpy(np.concatenate(parts)).cuda()
    with kc.Counter(k=ks[0]) as c:
        res = c.count_sets(buf.data_ptr(), sets)
        low_all, (roots_all, _) = c.low_bytes(), c.root_records()
        for (o, n, k), r, d in zip(sets, res, datas):
            low = oracle.unpack(low_all[r.low_offset:r.low_offset + r.low_bytes], k)
            rec = roots_all[r.root_offset:r.root_offset + r.root_records]
            parity.check_layout(low, rec, list(r.root_counts), k)
            mk, mc = parity.merged(low, rec, k)
            keys, counts, K = oracle.count(d, k)
            assert r.total_kmers == K and np.array_equal(mk, keys) and np.array_equal(mc, counts.astype(np.uint64))
