"""Restarting a resident stream without waits, beyond host appends of a plain
array: device appends ordered by the producer's stream, pyramids whose append
dim folds, arrays of several lengths one after the other; and a server whose
resident stream had a request that failed."""
import ctypes as C

import pytest
import torch

import cases
import chucky_gb300 as cg
import harness as H
import test_failures as F
from chucky_gb300 import capi

pytestmark = pytest.mark.gpu


def config(codec, fold):
    dims = capi.make_dims([dict(size=0, chunk=4, cps=2, name="t", downsample=fold),
                           dict(size=36, chunk=8, cps=2, name="y", downsample=1),
                           dict(size=64, chunk=16, cps=2, name="x", downsample=1)])
    cfg = capi.make_config(dims, dtype="u16", codec=codec, level=0 if codec == "none" else 1,
                           reduce="max", append_reduce="max", epochs_per_batch=2)
    cfg._dims = dims
    return cfg


@pytest.mark.parametrize("codec", ["none", "lz4", "zstd"])
@pytest.mark.parametrize("fold", [0, 1])
def test_device_appends(codec, fold):
    cfg = config(codec, fold)
    lib = cg.load()
    lib.tile_stream_gpu_restart.argtypes = [C.c_void_p, C.c_void_p]
    lib.tile_stream_gpu_append_device.restype = capi.WriterResult
    lib.tile_stream_gpu_append_device.argtypes = [C.c_void_p, capi.Slice, C.c_void_p]
    frame = 36 * 64
    data = cases.make_data("u16", 30 * frame, seed=11)
    host = torch.from_numpy(data.view("u1").copy()).pin_memory()
    buf = torch.zeros(7 * frame * 2, dtype=torch.uint8, device="cuda")
    side = torch.cuda.Stream()
    sink = H.MemSink()
    s = cg.GpuStream(cfg, sink.base)
    try:
        for turn, frames in enumerate((30, 8, 17, 1, 30)):
            if turn:
                sink.close()
                sink = H.MemSink()
                assert lib.tile_stream_gpu_restart(s.h, sink.base) == 0
            with torch.cuda.stream(side):
                for a in range(0, frames, 7):
                    n = (min(frames, a + 7) - a) * frame * 2
                    buf[:n].copy_(host[a * frame * 2:a * frame * 2 + n], non_blocking=True)
                    assert lib.tile_stream_gpu_append_device(
                        s.h, capi.Slice(buf.data_ptr(), buf.data_ptr() + n),
                        side.cuda_stream).error == 0
                    buf.zero_()  # (behind the stream's copy of it)
            assert s.flush().error == 0
            want, _ = (H.run_oracle(cfg, data[:frames * frame], quirks=False) if codec == "none"
                       else H.run_gpu(cfg, data[:frames * frame]))
            got = sink.shards()
            assert got == want, H.diff_shards(got, want)
    finally:
        s.close()
        sink.close()


@pytest.mark.parametrize("codec", ["none", "zstd"])
def test_server_after_a_failed_request(codec):
    from chucky_gb300 import serve
    cfg = config(codec, 1)
    data = cases.make_data("u16", 21 * 36 * 64, seed=12)
    dims = [dict(size=0, chunk=4, cps=2, name="t", downsample=1),
            dict(size=36, chunk=8, cps=2, name="y", downsample=1),
            dict(size=64, chunk=16, cps=2, name="x", downsample=1)]
    kw = dict(dtype="u16", codec=codec, level=0 if codec == "none" else 1, reduce="max",
              append_reduce="max", epochs_per_batch=2)
    want, _ = (H.run_oracle(cfg, data, quirks=False) if codec == "none" else H.run_gpu(cfg, data))
    with serve.Server(max_streams=1) as server:
        for fail, at in ((None, 1), ("write", 2), (None, 1), ("open", 3), (None, 1), (None, 1)):
            sink = H.MemSink() if fail is None else F.FaultySink(fail, at)
            r = serve.Request(name="a", cfg_kwargs=kw, dims=dims, data=data.view("u1"),
                              frame_bytes=36 * 64 * 2 * 5, sink=sink.base)
            if fail:
                with pytest.raises(RuntimeError):
                    server.replay([r], sink.base, paced=False)
                continue
            server.replay([r], sink.base, paced=False)
            got = sink.shards()
            sink.close()
            assert got == want, H.diff_shards(got, want)
