"""Element-wise transposes, one or four elements per thread, against the
oracle's bytes: even numbers of channels in chunks of their own, narrow and wide
chunk rows that are no multiple of 16 bytes, epochs that end inside a thread's
four elements."""
import pytest

import cases
import harness as H
import test_gpu_transpose as T
from chucky_gb300 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["u8", "u16", "f32", "f64"])
@pytest.mark.parametrize("channels,chunk_x", [(2, 15), (2, 17), (4, 7), (6, 15), (6, 17), (8, 5),
                                              (10, 17), (12, 25)])
def test_channels(dtype, channels, chunk_x):
    T.check(dtype, channels, 1, chunk_x, "c_before_yx", x=51)


@pytest.mark.parametrize("dtype", ["u8", "u16", "f32", "f64"])
@pytest.mark.parametrize("x,chunk_x", [(7, 1), (8, 1), (50, 7), (130, 63), (130, 65), (203, 100)])
@pytest.mark.parametrize("pos", [(0, 1, 2), (0, 2, 1)])
def test_rows(dtype, x, chunk_x, pos):
    dims = [dict(size=0, chunk=3, cps=2, name="t"), dict(size=5, chunk=2, cps=0, name="y"),
            dict(size=x, chunk=chunk_x, cps=0, name="x")]
    for d, p in zip(dims, pos):
        d["pos"] = p
    dims = capi.make_dims(dims)
    cfg = capi.make_config(dims, dtype=dtype, epochs_per_batch=1)
    n = int(2.4 * H.epoch_elements(cfg))
    data = cases.make_data(dtype, n, seed=x + chunk_x)
    a, _ = H.run_gpu(cfg, data)
    b, _ = H.run_oracle(cfg, data, quirks=False)
    assert a == b, H.diff_shards(a, b)
