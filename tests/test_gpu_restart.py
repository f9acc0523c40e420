"""A resident stream restarted for its next array (tile_stream_gpu_restart)
writes that array's shards as a new stream would: after a clean flush, and
after a sink that refused one batch and took the later ones, so that the flush
succeeds although the host's and the device's places in the shard differ."""
import ctypes as C

import pytest
import torch

import cases
import harness as H
import test_failures as F
from chucky_gb300 import capi

pytestmark = pytest.mark.gpu


def _restart(s, sink_base):
    lib = s.g.lib
    lib.tile_stream_gpu_restart.argtypes = [C.c_void_p, C.c_void_p]
    assert lib.tile_stream_gpu_restart(s.h, sink_base) == 0


@pytest.mark.parametrize("codec", ["none", "lz4"])
@pytest.mark.parametrize("fail", [None, "open", "write"])
def test_restart(fail, codec):
    dims = capi.make_dims([dict(size=0, chunk=1, cps=4, name="t"),
                           dict(size=24, chunk=8, cps=3, name="y"),
                           dict(size=64, chunk=16, cps=2, name="x")])
    cfg = capi.make_config(dims, dtype="u16", codec=codec, level=1, epochs_per_batch=2)
    frame = 24 * 64 * 2
    data = cases.make_data("u16", 6 * 24 * 64, seed=3).view("u1").reshape(-1)
    faulty = F.FaultySink(fail, 1)
    s = F.Stream("gpu", cfg, faulty.base)
    try:
        assert s.append(data, 0, 2 * frame)[0] == 0
        torch.cuda.synchronize()
        # the second batch's start delivers the first one, which is done
        error, _ = s.append(data, 2 * frame, 4 * frame)
        assert error == (1 if fail else 0)
        faulty.fail = None
        assert s.append(data, 4 * frame, 6 * frame)[0] == 0
        assert s.flush() == 0
        for n in (5, 6):  # a partly filled shard epoch, then a whole one and two more
            sink = H.MemSink()
            _restart(s, sink.base)
            assert s.append(data, 0, n * frame)[0] == 0
            assert s.flush() == 0
            got = sink.shards()
            sink.close()
            want, _ = H.run_gpu(cfg, data[:n * frame])
            assert got == want, H.diff_shards(got, want)
            if codec == "none":
                want, _ = H.run_oracle(cfg, data[:n * frame], quirks=False)
                assert got == want, H.diff_shards(got, want)
    finally:
        s.destroy()
