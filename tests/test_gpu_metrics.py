"""The aggregation metric holds the shard index of a batch whether the batch is
gathered beside it (below 1 MiB of chunks) or before it: two streams of nearly
the same size and the same index, one on each side of that line.  The index, a
checksum over 16 epochs of 65,536 entries, is most of the time."""
import numpy as np
import pytest

import chucky_gb300 as cg
import harness as H
from chucky_gb300 import capi

pytestmark = pytest.mark.gpu


def aggregate_ms(chunks):
    dims = capi.make_dims([dict(size=0, chunk=1, cps=16, name="t"),
                           dict(size=4 * chunks, chunk=4, cps=chunks, name="x")])
    cfg = capi.make_config(dims, dtype="f32", epochs_per_batch=1)
    data = np.zeros(16 * 4 * chunks, "<f4")
    best = 1e30
    for _ in range(3):
        sink = H.MemSink()
        s = cg.GpuStream(cfg, sink.base)
        H._drive(s.writer, data, None)
        m = s.metrics().aggregate
        assert m.count == 16
        best = min(best, m.ms)
        s.close()
        sink.close()
    return best


def test_index_is_in_the_aggregation():
    below, above = aggregate_ms(65535), aggregate_ms(65536)
    assert 0.75 * below < above, (below, above)
