"""The work whose speed is measured: what a program that ingests, encodes or
reads back chunked arrays has this library do, through its C entry points.

Three kinds of case:
  stream   an array appended to a resident tile_stream_gpu and flushed; the
           shard bytes come back.  The sink is a zero-copy one
           (shard_writer.write_direct): uncompressed shards are used where
           they are, in the stream's pinned delivery buffers (an array of at
           most two batches stays there until the next pass); compressed
           ones, whose size is not known beforehand, are put one after
           another into a store in device memory, for a later stage or a
           check by the device decoders, with asynchronous copies that the
           sink's fence waits for.
  serve    several arrays at once through a chucky_server (shared encoders).
  encode / decode   the batched chunk codecs on device memory.
Every output is bytes (compressed chunks, decoded chunks, shard contents), so
none has a value in 64 bits to be compared with: exact() gives None.
"""
import ctypes as C
import itertools

import numpy as np
import torch

import chucky_gb300
from chucky_gb300 import capi, serve

MIB = 1 << 20


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # one small camera snapshot stored uncompressed: launches, copies and
        # the host's path are all of it
        dict(name="stream_snapshot_u16", kind="stream", shape="txy", dtype="u16", data="sensor",
             t=1, y=256, x=256, ct=1, cy=64, cx=64, lod="", codec="none", level=0,
             reduce="mean", epochs=1, batch=1, host=True),
        # interleaved RGB video frames into planar chunks, sizes that chunks
        # do not divide: the element-wise transpose
        dict(name="stream_rgb_planar_u8", kind="stream", shape="rgb", dtype="u8", data="frames",
             t=4, y=1080, x=1919, ct=4, cy=256, cx=256, lod="", codec="none", level=0,
             reduce="mean", epochs=2, batch=1, host=False),
        # the 256^3 u16 cube from pinned host memory, LZ4, no pyramid
        dict(name="stream_cube_lz4", kind="stream", shape="zyx", dtype="u16", data="cube",
             t=64, y=256, x=256, ct=64, cy=64, cx=64, lod="", codec="lz4", level=1,
             reduce="mean", epochs=4, batch=2, host=True),
        # sensor frames 2304 x 4096 already on the device, (y, x) mean
        # pyramid, zstd-1: the acquisition stream at full rate
        dict(name="stream_sensor_pyramid_zstd", kind="stream", shape="tyx", dtype="u16",
             data="sensor", t=16, y=2304, x=4096, ct=16, cy=256, cx=256, lod="yx",
             codec="zstd", level=1, reduce="mean", epochs=2, batch=1, host=False),
        # 256^3 f32 volume, median pyramid in all three dims (the append dim
        # folds with a mean), uncompressed
        dict(name="stream_volume_f32_pyramid", kind="stream", shape="zyx", dtype="f32",
             data="smooth", t=64, y=256, x=256, ct=64, cy=64, cx=64, lod="tyx", codec="none",
             level=0, reduce="median", epochs=4, batch=2, host=False),
        # ragged volumes over time with more pyramid levels than a tile holds
        dict(name="stream_deep_pyramid_i16", kind="stream", shape="tzyx", dtype="i16",
             data="sensor", t=1, z=16, y=200, x=328, ct=1, cz=4, cy=16, cx=16, lod="zyx",
             codec="none", level=0, reduce="median", epochs=2, batch=1, host=False),
        # four arrays of different shapes, types and codecs ingested at once
        dict(name="serve_four_arrays", kind="serve", cube=4, sensor=16, stack=2, frames8=128),
        # an acquisition loop's encoder call that allocates nothing, on a few
        # small chunks
        dict(name="encode_lz4_static_small", kind="encode", codec="lz4", level=1, data="frames",
             chunk=16384, n=16, static=True),
        # a batch of 32 x 256 x 256 u16 sensor chunks: LZ4 at its default level
        dict(name="encode_lz4_sensor", kind="encode", codec="lz4", level=1, data="sensor",
             chunk=4 * MIB, n=64, static=False),
        # the cube's 64^3 chunks at zstd level 3: the wide match window
        dict(name="encode_zstd3_cube", kind="encode", codec="zstd", level=3, data="cube",
             chunk=MIB // 2, n=64, static=False),
        # reading stores back on the device: sensor chunks in LZ4 ...
        dict(name="decode_lz4_sensor", kind="decode", codec="lz4", level=1, data="sensor",
             chunk=MIB, n=64),
        # ... and the cube's chunks in zstd
        dict(name="decode_zstd_cube", kind="decode", codec="zstd", level=3, data="cube",
             chunk=MIB // 2, n=64),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["stream", "stream", "encode", "decode"])
    if kind == "stream":
        dtype = rng.choice(["u8", "u16", "i16", "f16", "f32", "u32"])
        data = "frames" if dtype == "u8" else "stack" if dtype[0] == "f" else "sensor"
        codec, level = rng.choice([("none", 0), ("lz4", 1), ("zstd", 1), ("zstd", 3)])
        ct = rng.choice([1, 4, 16, 32])
        y, x = _log(rng, 64, 2304), _log(rng, 64, 2304)
        while ct * y * x > 16 << 20:  # frames of one epoch
            y = max(64, y // 2)
        # the append dim's pyramid drains at the flush, a batch of its own
        lod = rng.choice(["", "yx", "tyx"]) if ct > 1 else rng.choice(["", "yx"])
        edge = rng.choice([32, 64, 100, 128])
        return dict(kind="stream", shape="tyx", dtype=dtype, data=data, t=ct, y=y, x=x, ct=ct,
                    cy=edge, cx=rng.choice([edge, 2 * edge]), lod=lod, codec=codec, level=level,
                    reduce=rng.choice(["mean", "min", "max", "median", "max_sup", "min_sup"]),
                    epochs=1 if lod == "tyx" else rng.choice([1, 2]), batch=1,
                    host=rng.random() < 0.5)
    codec = rng.choice(["lz4", "zstd"])
    level = rng.choice([1, 1, 2 if codec == "lz4" else 3])
    data = rng.choice(["sensor", "cube", "frames", "stack", "mix"])
    chunk = _log(rng, 4096, 4 * MIB if kind == "encode" else MIB)
    total = _log(rng, MIB // 4, 128 * MIB if kind == "encode" and level == 1 else 32 * MIB)
    c = dict(kind=kind, codec=codec, level=level, data=data, chunk=chunk,
             n=max(1, min(4096, total // chunk)))
    if kind == "encode":
        c["static"] = False
    return c


# compressed bytes per input byte of the data below (what an encoder cannot
# do without writing), by measurement
_RATIO = {("lz4", "sensor"): 0.81, ("lz4", "cube"): 1.0, ("lz4", "frames"): 1.0,
          ("lz4", "stack"): 1.0, ("lz4", "mix"): 0.26, ("lz4", "smooth"): 1.0,
          ("zstd", "sensor"): 0.5, ("zstd", "cube"): 0.66, ("zstd", "frames"): 0.76,
          ("zstd", "stack"): 0.93, ("zstd", "mix"): 0.26, ("zstd", "smooth"): 0.9}


def work(case):
    if case["kind"] == "serve":
        n = (case["cube"] * 64 * 256 * 256 * 2 * (1 + 1.0)
             + case["sensor"] * 2304 * 4096 * 2 * (1 + 0.5 * 4 / 3)
             + case["stack"] * 64 * 512 * 512 * 4 * (1 + 1.0)
             + case["frames8"] * 1024 * 1024 * (1 + 0.76 * 4 / 3))
        return {"bytes": n, "flops": 0}
    if case["kind"] == "stream":
        n = (case["epochs"] * case["t"] * case.get("z", 1) * case["y"] * case["x"]
             * (3 if case["shape"] == "rgb" else 1) * capi.BPE[case["dtype"]])
        out = {0: 1.0, 2: 4 / 3, 3: 8 / 7}[len(case["lod"])]
        return {"bytes": n * (1 + out * _RATIO.get((case["codec"], case["data"]), 1.0)),
                "flops": 0}
    n = case["chunk"] * case["n"]
    return {"bytes": n * (1 + _RATIO[case["codec"], case["data"]]), "flops": 0}


def exact(case, seed):
    return None


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


_TORCH = {"u8": torch.uint8, "u16": torch.int16, "i16": torch.int16, "u32": torch.int32,
          "f16": torch.float16, "f32": torch.float32}


def _values(data, dtype, n, chunk, g):
    """n values of `dtype` on the device: detector counts ("sensor": Poisson
    with brighter spots, 12 bits), a textured volume ("cube"), 6-bit frames
    ("frames"), noise ("stack"), a smooth field with noise ("smooth"), or
    chunks of `chunk` values that are zero, constant or random ("mix")."""
    dev = "cuda"
    if data == "sensor":
        v = torch.poisson(torch.full((min(n, 1 << 24),), 100.0, device=dev), generator=g)
        if v.numel() < n:  # larger inputs: rolled repeats farther apart than any window
            v = torch.cat([torch.roll(v, 7919 * k) for k in range(-(-n // v.numel()))])[:n]
        spots = torch.randint(0, max(1, n - 64), (max(1, n // 4096),), device=dev, generator=g)
        for k in range(16):
            v[spots + k] += 40.0 * k
        v = v.clamp_(max=255.0 if dtype == "u8" else 4095.0)
    elif data == "cube":
        e = torch.arange(n, device=dev, dtype=torch.int64)
        c, e = e // max(1, chunk), e % max(1, chunk)
        v = ((e % 64) ^ ((e // 64) % 64) ^ ((e // 4096 + 64 * c) % 256)) * 257
        v = (v + torch.randint(0, 16, (n,), device=dev, generator=g)) % 65536
        v = torch.where(v >= 32768, v - 65536, v) if dtype in ("u16", "i16") else v
    elif data == "frames":
        v = torch.randint(0, 64, (n,), device=dev, generator=g, dtype=torch.uint8)
    elif data == "stack":
        v = torch.randn(n, device=dev, generator=g)
    elif data == "smooth":
        e = torch.arange(n, device=dev, dtype=torch.float32)
        v = torch.sin(e * 0.003) * torch.cos(e * 0.00002)
        v = v + 0.01 * torch.randn(n, device=dev, generator=g)
    else:
        k = -(-n // chunk)
        cls = torch.rand(k, device=dev, generator=g)
        const = torch.randint(1, 100, (k,), device=dev, generator=g)
        r = torch.randint(-(1 << 15), 1 << 15, (k, chunk), device=dev, generator=g,
                          dtype=torch.int32)
        v = torch.where((cls < 0.75)[:, None], const[:, None].to(torch.int32), r)
        v = torch.where((cls < 0.5)[:, None], torch.zeros_like(v), v).reshape(-1)[:n]
    return v.to(_TORCH[dtype])


_DTYPE_OF = {"sensor": "u16", "cube": "u16", "frames": "u8", "stack": "f32", "smooth": "f32",
             "mix": "u16"}


def _chunks(case, seed):
    """(n, stride) device bytes of a codec case, stride a multiple of 16 and
    256 readable bytes past the last chunk."""
    dtype = _DTYPE_OF[case["data"]]
    per = -(-case["chunk"] // capi.BPE[dtype])
    v = _values(case["data"], dtype, per * case["n"], per, _gen(seed))
    v = v.view(torch.uint8).reshape(case["n"], -1)[:, :case["chunk"]]
    stride = (case["chunk"] + 15) // 16 * 16
    buf = torch.zeros(case["n"] * stride + 256, dtype=torch.uint8, device="cuda")
    buf[:case["n"] * stride].view(case["n"], stride)[:, :case["chunk"]] = v
    return buf, stride


# ---------------------------------------------------------------------------
# a zero-copy sink (include/writer.h)
# ---------------------------------------------------------------------------

_WRITE = C.CFUNCTYPE(C.c_int, C.c_void_p, C.c_uint64, C.c_void_p, C.c_void_p)
_FINAL = C.CFUNCTYPE(C.c_int, C.c_void_p)
_OPEN = C.CFUNCTYPE(C.c_void_p, C.c_void_p, C.c_uint8, C.c_uint64)
_WAIT = C.CFUNCTYPE(None, C.c_void_p, C.c_uint8, C.c_uint64)  # io_event: one u64


class _ShardWriter(C.Structure):
    _fields_ = [("write", _WRITE), ("write_direct", _WRITE), ("finalize", _FINAL),
                ("sink", C.c_uint64), ("level", C.c_uint64), ("shard", C.c_uint64)]


class _ShardSink(C.Structure):
    _fields_ = [("open", _OPEN), ("update_append", C.c_void_p), ("record_fence", C.c_void_p),
                ("wait_fence", _WAIT), ("id", C.c_uint64)]


_sinks = {}
_ids = itertools.count(1)


def _where(w):
    o = _ShardWriter.from_address(w)
    return _sinks[o.sink], (o.level, o.shard)


@_WRITE
def _write(w, offset, beg, end):
    s, key = _where(w)
    s.small.append((key, offset, C.string_at(beg, end - beg)))
    return 0


@_WRITE
def _write_direct(w, offset, beg, end):
    s, key = _where(w)
    s.put(key, offset, beg, end - beg)
    return 0


@_FINAL
def _finalize(w):
    return 0


@_OPEN
def _open(sink, level, shard):
    s = _sinks[_ShardSink.from_address(sink).id]
    w = s.writers.get((level, shard))
    if w is None:
        w = _ShardWriter(_write, _write_direct, _finalize, s.id, level, shard)
        s.writers[level, shard] = w
    return C.addressof(w)


@_WAIT
def _wait(sink, level, event):
    _sinks[_ShardSink.from_address(sink).id].wait()


class _View:
    """Bytes of a buffer that `owner` keeps alive, for np.asarray."""

    def __init__(self, ptr, n, owner):
        self.__array_interface__ = {"shape": (n,), "typestr": "|u1", "data": (ptr, False),
                                    "version": 3}
        self.owner = owner


class _Sink:
    """`store_bytes`: the capacity of the device store; 0 keeps the pieces
    where they are delivered."""

    def __init__(self, store_bytes=0):
        self.id = next(_ids)
        self.writers, self.small, self.large, self.used, self.busy = {}, [], [], 0, False
        self.store = self.side = None
        if store_bytes:
            self.store = torch.zeros(store_bytes, dtype=torch.uint8, device="cuda")
            self.side = torch.cuda.Stream()
        self.base = _ShardSink(_open, None, None, _wait if store_bytes else _WAIT(), self.id)
        self.ptr = C.addressof(self.base)
        _sinks[self.id] = self

    def clear(self):
        self.small, self.large, self.used = [], [], 0

    def put(self, key, offset, ptr, n):
        self.large.append((key, offset, ptr, n))
        if self.store is not None:
            src = torch.from_numpy(np.asarray(_View(ptr, n, self)))
            with torch.cuda.stream(self.side):
                self.store[self.used:self.used + n].copy_(src, non_blocking=True)
            self.used += n
            self.busy = True

    def wait(self):
        if self.busy:
            self.side.synchronize()
            self.busy = False

    def shards(self, owner):
        """The shards' data (the store, or the pieces in order), and their
        index blobs in one."""
        index = np.frombuffer(b"".join(b for _, _, b in sorted(self.small)), dtype=np.uint8)
        if self.store is not None:
            return self.store, index
        return [np.asarray(_View(p, n, owner)) for _, _, p, n in sorted(self.large)], index

    def close(self):
        _sinks.pop(self.id, None)


# ---------------------------------------------------------------------------
# streams
# ---------------------------------------------------------------------------

def _dims(case):
    D, lod = dict, case["lod"]
    z = [D(size=case["z"], chunk=case["cz"], cps=0, name="z")] if case["shape"] == "tzyx" else []
    c = [D(size=3, chunk=1, cps=3, name="c")] if case["shape"] == "rgb" else []
    dims = ([D(size=0, chunk=case["ct"], cps=1, name="t")] + z
            + [D(size=case["y"], chunk=case["cy"], cps=0, name="y"),
               D(size=case["x"], chunk=case["cx"], cps=0, name="x")] + c)
    for d in dims:
        d["downsample"] = 1 if d["name"] in lod else 0
    if c:  # t, y, x, c in memory; t, c, y, x in storage
        for d, pos in zip(dims, (0, 2, 3, 1)):
            d["pos"] = pos
    return dims


def _bind(lib):
    P = C.c_void_p
    lib.tile_stream_gpu_restart.argtypes = [P, P]
    lib.tile_stream_gpu_append_device.restype = capi.WriterResult
    lib.tile_stream_gpu_append_device.argtypes = [P, capi.Slice, P]
    lib.chucky_encode_scratch_bytes.restype = C.c_size_t
    lib.chucky_encode_scratch_bytes.argtypes = [C.c_int, C.c_int, C.c_size_t, C.c_size_t]
    lib.chucky_encode_bound.restype = C.c_size_t
    lib.chucky_encode_bound.argtypes = [C.c_int, C.c_size_t]
    lib.chucky_encode_chunks.argtypes = [C.c_int, C.c_int, P, C.c_size_t, C.c_size_t, C.c_size_t,
                                         P, C.c_size_t, P, P, C.c_size_t, P]
    lib.chucky_lz4_encode_chunks_static.argtypes = [P, C.c_size_t, C.c_size_t, C.c_size_t, P,
                                                    C.c_size_t, P, P]
    for f in (lib.chucky_lz4_decode_chunks, lib.chucky_zstd_decode_chunks):
        f.argtypes = [P, P, P, C.c_size_t, P, C.c_size_t, C.c_size_t, P, P]
    return capi.bind_server(lib)


def _capacity(lib, cfg, epochs):
    """Bytes that `epochs` epochs and the flush's drain can come to."""
    info = capi.MemoryInfo()
    if lib.tile_stream_gpu_memory_estimate(C.byref(cfg), C.byref(info)):
        raise RuntimeError("invalid configuration")
    return (epochs + 1) * info.total_chunks * info.max_output_size


class _Stream:
    """A resident stream, its input and its sink."""

    def __init__(self, case, seed):
        self.lib = _bind(chucky_gb300.load())
        self.dims = capi.make_dims(_dims(case))
        self.cfg = capi.make_config(
            self.dims, dtype=case["dtype"], codec=case["codec"], level=case["level"],
            reduce=case["reduce"], epochs_per_batch=case["batch"],
            max_nlod=0 if case["shape"] == "tzyx" else 4, buffer_capacity_bytes=32 * MIB)
        n = (case["epochs"] * case["t"] * case.get("z", 1) * case["y"] * case["x"]
             * (3 if case["shape"] == "rgb" else 1))
        self.sink = _Sink(0 if case["codec"] == "none" else _capacity(self.lib, self.cfg, case["epochs"]))
        self.gpu = chucky_gb300.GpuStream(self.cfg, self.sink.ptr)
        v = _values(case["data"], case["dtype"], n, 64 ** 3, _gen(seed)).view(torch.uint8)
        self.host = case["host"]
        self.input = v.cpu().pin_memory() if self.host else v
        self.side = None if self.host else torch.cuda.Stream()
        step = n * capi.BPE[case["dtype"]] // case["epochs"]  # an append per epoch
        p = self.input.data_ptr()
        self.slices = [capi.Slice(p + k * step, p + (k + 1) * step)
                       for k in range(case["epochs"])]

    def run(self):
        self.sink.clear()
        if self.lib.tile_stream_gpu_restart(self.gpu.h, None):
            raise RuntimeError("restart failed")
        for s in self.slices:
            if self.host:
                r = self.lib.writer_append(self.gpu.writer, s)
            else:
                r = self.lib.tile_stream_gpu_append_device(self.gpu.h, s, self.side.cuda_stream)
            if r.error:
                raise RuntimeError("append failed")
        if self.gpu.flush().error:
            raise RuntimeError("flush failed")
        return self.sink.shards(self)

    def __del__(self):
        if hasattr(self, "gpu"):
            self.gpu.close()
        if hasattr(self, "sink"):
            self.sink.close()


class _Serve:
    """A server with resident streams and the requests it is given at once:
    a cube in LZ4, sensor frames with a pyramid in zstd, f32 stacks in LZ4,
    8-bit frames with a pyramid in zstd."""

    def __init__(self, case, seed):
        _bind(chucky_gb300.load())
        D = dict
        g = _gen(seed)
        spec = [
            ("cube", "u16", "cube", case["cube"] * 64 * 256 * 256, 256 * 256 * 2 * 64, 2,
             dict(codec="lz4"), [D(size=0, chunk=64, cps=4, name="z"),
                                 D(size=256, chunk=64, cps=4, name="y"),
                                 D(size=256, chunk=64, cps=4, name="x")]),
            ("sensor", "u16", "sensor", case["sensor"] * 2304 * 4096, 2304 * 4096 * 2, 1,
             dict(codec="zstd", max_nlod=4),
             [D(size=0, chunk=16, cps=1, name="t"),
              D(size=2304, chunk=256, cps=0, name="y", downsample=1),
              D(size=4096, chunk=256, cps=0, name="x", downsample=1)]),
            ("stack", "f32", "stack", case["stack"] * 64 * 512 * 512, 64 * 512 * 512 * 4, 1,
             dict(codec="lz4"), [D(size=0, chunk=1, cps=1, name="t"),
                                 D(size=64, chunk=64, cps=1, name="z"),
                                 D(size=512, chunk=128, cps=0, name="y"),
                                 D(size=512, chunk=128, cps=0, name="x")]),
            ("frames8", "u8", "frames", case["frames8"] * 1024 * 1024, 1024 * 1024 * 8, 1,
             dict(codec="zstd", max_nlod=4),
             [D(size=0, chunk=64, cps=1, name="t"),
              D(size=1024, chunk=256, cps=0, name="y", downsample=1),
              D(size=1024, chunk=256, cps=0, name="x", downsample=1)]),
        ]
        self.sinks, self.requests, self.lib = [], [], chucky_gb300.load()
        for name, dtype, data, n, append, batch, kw, dims in spec:
            v = _values(data, dtype, n, 64 ** 3, g).view(torch.uint8)
            kw = dict(dtype=dtype, level=1, epochs_per_batch=batch, **kw)
            r = serve.Request(name=name, cfg_kwargs=kw, dims=dims, data=v, frame_bytes=append)
            epochs = -(-n // (dims[0]["chunk"] * int(np.prod([d["size"] for d in dims[1:]]))))
            self.sinks.append(_Sink(_capacity(self.lib, r.config(), epochs)))
            r.sink = self.sinks[-1].ptr
            self.requests.append(r)
        self.server = serve.Server(max_streams=len(spec))
        self.server.prewarm(self.requests, self.sinks[0].ptr)

    def run(self):
        for s in self.sinks:
            s.clear()
        self.server.replay(self.requests, self.sinks[0].ptr, paced=False)
        return {r.name: s.shards(self) for r, s in zip(self.requests, self.sinks)}

    def __del__(self):
        if hasattr(self, "server"):
            self.server.close()
        for s in getattr(self, "sinks", []):
            s.close()


# ---------------------------------------------------------------------------
# codecs
# ---------------------------------------------------------------------------

class _Encode:
    def __init__(self, case, seed):
        self.lib, self.case = _bind(chucky_gb300.load()), case
        self.codec = capi.CODEC[case["codec"]]
        self.buf, self.stride = _chunks(case, seed)
        bound = self.lib.chucky_encode_bound(self.codec, case["chunk"])
        self.out_stride = (bound + 15) // 16 * 16
        self.out = torch.zeros((case["n"], self.out_stride), dtype=torch.uint8, device="cuda")
        self.sizes = torch.zeros(case["n"], dtype=torch.int64, device="cuda")
        self.scratch_bytes = 0 if case["static"] else self.lib.chucky_encode_scratch_bytes(
            self.codec, case["level"], case["chunk"], case["n"])
        self.scratch = torch.empty(max(16, self.scratch_bytes), dtype=torch.uint8, device="cuda")

    def run(self):
        c, st = self.case, torch.cuda.current_stream().cuda_stream
        if c["static"]:
            rc = self.lib.chucky_lz4_encode_chunks_static(
                self.buf.data_ptr(), c["chunk"], self.stride, c["n"], self.out.data_ptr(),
                self.out_stride, self.sizes.data_ptr(), st)
        else:
            rc = self.lib.chucky_encode_chunks(
                self.codec, c["level"], self.buf.data_ptr(), c["chunk"], self.stride, c["n"],
                self.out.data_ptr(), self.out_stride, self.sizes.data_ptr(),
                self.scratch.data_ptr(), self.scratch_bytes, st)
        if rc:
            raise RuntimeError("encode failed")
        return {"chunks": self.out, "sizes": self.sizes}


class _Decode:
    """Encoded chunks packed one after another, as a shard holds them."""

    def __init__(self, case, seed):
        e = _Encode(dict(case, static=False), seed)
        r = e.run()
        sizes = r["sizes"].cpu()
        self.blob = torch.cat([r["chunks"][i, :k] for i, k in enumerate(sizes.tolist())])
        self.lib, self.case = e.lib, case
        self.sizes = sizes.cuda()
        self.offsets = (torch.cumsum(sizes, 0) - sizes).cuda()
        self.out = torch.zeros((case["n"], case["chunk"]), dtype=torch.uint8, device="cuda")
        self.status = torch.zeros(case["n"], dtype=torch.int32, device="cuda")
        self.call = (self.lib.chucky_lz4_decode_chunks if case["codec"] == "lz4"
                     else self.lib.chucky_zstd_decode_chunks)

    def run(self):
        c = self.case
        if self.call(self.blob.data_ptr(), self.offsets.data_ptr(), self.sizes.data_ptr(), c["n"],
                     self.out.data_ptr(), c["chunk"], c["chunk"], self.status.data_ptr(),
                     torch.cuda.current_stream().cuda_stream):
            raise RuntimeError("decode failed")
        return {"chunks": self.out, "status": self.status}


_KINDS = {"stream": _Stream, "serve": _Serve, "encode": _Encode, "decode": _Decode}


def prepare(case, seed):
    return _KINDS[case["kind"]](case, seed)


def run(state):
    return state.run()
