"""A streamed count leaves its first occurrences with the sink: calls that read
them afterwards are refused (they read from a null pointer before), the root
records stay, and the next count on the context is whole again."""
import numpy as np
import pytest

import kmertreecounter_b200 as kc
import parity
from kmertreecounter_b200 import sizing, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [31, 63, 101])
def test_calls_after_a_streamed_count(tmp_path, k):
    data = synth.fastq(synth.params(seed=k, genome_len=40_000, n_reads=3000, read_len=(120, 150)))
    with kc.Counter(k=k) as c:
        st = c.count_host_stream(data.ctypes.data, data.size, lambda kind, root, addr, n: 0)
        assert st.low_records > 0 and st.root_records > 0
        for call in (lambda: c.histogram(1, 100), lambda: sizing.bucket_loads(c), c.low_bytes,
                     lambda: c.post_process(str(tmp_path))):
            with pytest.raises(kc.KcError) as e:
                call()
            assert e.value.code == kc.KC_ERR_STATE
        roots, _ = c.root_records()
        assert roots.shape[0] == st.root_records
        c.count_host(data)
        parity.check_exact(c, data, k)
        assert int(np.sum(c.histogram(1, 5000)[0])) > 0
