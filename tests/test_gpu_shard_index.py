"""Shard index checksums at the sizes where the index kernel's split of the
index among its 256 threads changes: a shard of one chunk, of fewer index
words than threads, exactly as many, one chunk more, and several words per
thread; with and without page-aligned shards, several shards and shard epochs
(the file's crc32c and offsets compared byte for byte with the oracle's)."""
import pytest

import cases
import harness as H
from chucky_gb300 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("alignment", [0, 512])
@pytest.mark.parametrize("chunks", [1, 2, 127, 128, 129, 1025])
def test_index_bytes(chunks, alignment):
    dims = capi.make_dims([dict(size=0, chunk=1, cps=2, name="t"),
                           dict(size=6, chunk=3, cps=1, name="y"),
                           dict(size=4 * chunks, chunk=4, cps=chunks, name="x")])
    cfg = capi.make_config(dims, dtype="u16", epochs_per_batch=2, shard_alignment=alignment)
    data = cases.make_data("u16", 5 * 6 * 4 * chunks, seed=chunks)
    a, _ = H.run_gpu(cfg, data)
    b, _ = H.run_oracle(cfg, data, quirks=False)
    assert a == b, H.diff_shards(a, b)
