"""Streams without a codec and the device copies of their delivery slots (from 1
MiB of chunks per batch on): they do without them where a budget or the device
has no room, and what was accepted with a budget stays accepted.  With and
without them, aligned shards and partial batches included, the shards are the
oracle's."""
import ctypes as C

import numpy as np
import pytest

import cases
import chucky_gb300 as cg
import harness as H
from chucky_gb300 import capi

MIB = 1 << 20


def config(t=8, y=256, x=256, dtype="f32", chunk=64, batch=2, lod=0, **kw):
    dims = capi.make_dims([dict(size=0, chunk=t, cps=2, name="t"),
                           dict(size=y, chunk=chunk, cps=2, name="y", downsample=lod),
                           dict(size=x, chunk=chunk, cps=2, name="x", downsample=lod)])
    cfg = capi.make_config(dims, dtype=dtype, epochs_per_batch=batch, **kw)
    cfg._dims = dims
    return cfg


def estimate(cfg):
    info = capi.MemoryInfo()
    assert cg.load().tile_stream_gpu_memory_estimate(C.byref(cfg), C.byref(info)) == 0
    return info


def copies(cfg):
    """Bytes of the two slots' copies (no alignment)."""
    i = estimate(cfg)
    return 2 * (i.epochs_per_batch * i.total_chunks * i.max_output_size + 64)


def test_copies_are_counted():
    for cfg, least in ((config(), 6.1 * MIB), (config(codec="lz4", level=1), 8 * MIB)):
        assert estimate(cfg).device_bytes > least + copies(cfg)


@pytest.mark.parametrize("t,batch", [(8, 2), (16, 1), (4, 8)])
def test_advice_keeps_its_chunk_sizes(t, batch):
    """The largest chunk whose stream fits the budget without the copies."""
    cfg = config(t=t, batch=batch)
    ratios = (C.c_uint8 * 3)(1, 1, 1)
    lib = cg.load()
    target = 64 << 10
    assert lib.tile_stream_gpu_advise_chunk_sizes(C.byref(cfg), target, ratios, 1 << 40) == 0
    want = [d.chunk_size for d in cfg._dims]
    assert int(np.prod(want)) * 4 == target
    need = estimate(cfg).device_bytes - copies(cfg)
    assert lib.tile_stream_gpu_advise_chunk_sizes(C.byref(cfg), target, ratios, need) == 0
    assert [d.chunk_size for d in cfg._dims] == want
    assert lib.tile_stream_gpu_advise_chunk_sizes(C.byref(cfg), target, ratios, need - 1) == 0
    assert int(np.prod([d.chunk_size for d in cfg._dims])) * 4 < target


def data_of(cfg, epochs, seed):
    return cases.make_data("f32", int(epochs * H.epoch_elements(cfg)), seed=seed)


@pytest.mark.gpu
@pytest.mark.parametrize("alignment", [0, 512, 4096])
@pytest.mark.parametrize("epochs,lod", [(5.3, 0), (6, 0), (5.3, 1)])
def test_large_batches(epochs, lod, alignment):
    """5.3 epochs: whole batches, then one of an epoch and a part of one."""
    cfg = config(y=200, x=300, lod=lod, reduce="mean", max_nlod=3 if lod else 0,
                 shard_alignment=alignment)
    data = data_of(cfg, epochs, 7)
    want, _ = H.run_oracle(cfg, data, quirks=False)
    got, _ = H.run_gpu(cfg, data)
    assert got == want, H.diff_shards(got, want)


@pytest.mark.gpu
def test_device_without_room():
    """Room for the stream and half of its copies: it is made without them."""
    import torch
    cfg = config(t=64, y=512, x=512)
    data = data_of(cfg, 2.2, 8)
    want, _ = H.run_oracle(cfg, data, quirks=False)
    got, _ = H.run_gpu(cfg, data[:64 * 512 * 512])  # (loads the kernels)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    info, extra = estimate(cfg), copies(cfg)
    need = info.device_bytes - extra + info.shard_bytes + 64 * MIB
    hold = torch.empty(torch.cuda.mem_get_info()[0] - (need + extra // 2), dtype=torch.uint8,
                       device="cuda")
    try:
        got, _ = H.run_gpu(cfg, data)
    finally:
        del hold
        torch.cuda.empty_cache()
    assert got == want, H.diff_shards(got, want)


@pytest.mark.gpu
@pytest.mark.parametrize("budget", ["least", "some", "all"])
@pytest.mark.parametrize("lod", [0, 1])
def test_server(budget, lod):
    """A budget for one stream without copies, for two (admitted one at a time
    or together, never with copies), and for all with copies."""
    from chucky_gb300 import serve
    n = 3
    kw = dict(dtype="f32", epochs_per_batch=2, reduce="mean", max_nlod=3 if lod else 0)
    dims = [dict(size=0, chunk=8, cps=2, name="t"),
            dict(size=200, chunk=64, cps=2, name="y", downsample=lod),
            dict(size=300, chunk=64, cps=2, name="x", downsample=lod)]
    sinks = [H.MemSink() for _ in range(n)]
    try:
        reqs = []
        for i, s in enumerate(sinks):
            cfg = config(y=200, x=300, lod=lod, reduce="mean", max_nlod=3 if lod else 0)
            data = data_of(cfg, 4.6 + i, i)
            reqs.append(serve.Request(name=str(i), cfg_kwargs=kw, dims=dims, data=data.view("u1"),
                                      frame_bytes=8 * 200 * 300 * 4 // 2, sink=s.base))
        full = serve.memory_estimate(reqs[0])
        hbm = {"least": full - copies(reqs[0].config()), "some": 2 * full - 1, "all": 64 * full}[budget]
        st = serve.run_served(reqs, hbm_budget=hbm, max_streams=2, paced=False, warmup=False)
        assert st["requests"] == n
        for i, s in enumerate(sinks):
            cfg = config(y=200, x=300, lod=lod, reduce="mean", max_nlod=3 if lod else 0)
            want, _ = H.run_oracle(cfg, data_of(cfg, 4.6 + i, i), quirks=False)
            got = s.shards()
            assert got == want, H.diff_shards(got, want)
    finally:
        for s in sinks:
            s.close()
