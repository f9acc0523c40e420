"""Streams without a pyramid whose innermost dim is narrow or moves in
storage, against the oracle's bytes: every number of interleaved channels
around those the planar kernel takes (2 to 4), whole and split over chunks,
every element width, chunk rows that are and are not a multiple of 16 bytes,
array sizes that chunks do not divide, and storage orders that put the
channels first, between, or last."""
import pytest

import cases
import harness as H
from chucky_gb300 import capi

pytestmark = pytest.mark.gpu

# storage position of (t, y, x, c)
ORDERS = {"c_before_yx": (0, 2, 3, 1), "c_between": (0, 1, 3, 2), "c_last": (0, 1, 2, 3),
          "x_before_y": (0, 3, 2, 1)}


def check(dtype, channels, chunk_c, chunk_x, order, x=50):
    dims = [dict(size=0, chunk=2, cps=2, name="t"), dict(size=7, chunk=3, cps=0, name="y"),
            dict(size=x, chunk=chunk_x, cps=0, name="x"),
            dict(size=channels, chunk=chunk_c, cps=0, name="c")]
    for d, pos in zip(dims, ORDERS[order]):
        d["pos"] = pos
    dims = capi.make_dims(dims)
    cfg = capi.make_config(dims, dtype=dtype, epochs_per_batch=1)
    n = int(2.5 * H.epoch_elements(cfg))
    data = cases.make_data(dtype, n, seed=channels + chunk_x)
    a, _ = H.run_gpu(cfg, data)
    b, _ = H.run_oracle(cfg, data, quirks=False)
    assert a == b, H.diff_shards(a, b)


@pytest.mark.parametrize("order", list(ORDERS))
@pytest.mark.parametrize("dtype", ["u8", "u16", "f32", "f64"])
@pytest.mark.parametrize("channels,chunk_c", [(1, 1), (2, 1), (2, 2), (3, 1), (3, 3), (3, 2),
                                              (4, 1), (4, 2), (5, 1)])
def test_channels(dtype, channels, chunk_c, order):
    check(dtype, channels, chunk_c, 16, order)


@pytest.mark.parametrize("dtype", ["u8", "u16", "f32", "f64"])
@pytest.mark.parametrize("chunk_x", [1, 2, 4, 8, 12, 24, 48])
def test_chunk_rows(dtype, chunk_x):
    check(dtype, 3, 1, chunk_x, "c_before_yx")


@pytest.mark.parametrize("x", [16, 340, 700, 3000, 6000])
def test_row_tables(x):
    # rows of the offset tables: the channels alone, with x, with x and y
    check("u8", 3, 1, 16, "c_before_yx", x=x)
