"""The block-parallel zstd decoder against the sequential one, which decodes
the same calls while a stream is captured (no scratch can be had then): frames
of libzstd at fast, default and high levels (repeat offsets, tables per block,
RLE and raw blocks, 128 KiB blocks) and of this library's encoder, chunks
around the block, tile and thread-count edges, every output alignment; the
same frames cut short or with a byte changed, several frames, skippable ones.
Statuses and the bytes of whole chunks must be the same."""
import ctypes as C

import numpy as np
import pytest

from chucky_gb300 import load

pytestmark = pytest.mark.gpu


def data(kind, n, seed):
    rng = np.random.default_rng(seed)
    if kind == "poisson":
        return rng.poisson(30, n).astype(np.uint8)
    if kind == "text":  # words: many short matches and repeat offsets
        words = [rng.integers(97, 123, int(k), dtype=np.uint8).tobytes() + b" "
                 for k in rng.integers(2, 9, 300)]
        b = b"".join(words[int(k)] for k in rng.integers(0, 300, n // 3 + 2))
        return np.frombuffer(b[:n], np.uint8).copy()
    if kind == "rows":  # repeated records with a few changes: long matches
        row = rng.integers(0, 256, 700, dtype=np.uint8)
        x = np.resize(row, n)
        x[rng.integers(0, n, max(1, n // 300))] ^= 1
        return x
    if kind == "runs":
        return np.repeat(rng.integers(0, 4, n // 50 + 1, dtype=np.uint8), 50)[:n]
    x = rng.integers(0, 256, n, dtype=np.uint8)  # raw, RLE and coded blocks
    x[n // 3:n // 2] = 7
    x[n // 2:] &= 15
    return x


def compress(x, level):
    z = C.CDLL("libzstd.so.1")
    z.ZSTD_compressBound.restype = z.ZSTD_compress.restype = C.c_size_t
    z.ZSTD_compressBound.argtypes = [C.c_size_t]
    z.ZSTD_compress.argtypes = [C.c_char_p, C.c_size_t, C.c_char_p, C.c_size_t, C.c_int]
    cap = z.ZSTD_compressBound(len(x))
    buf = C.create_string_buffer(cap)
    k = z.ZSTD_compress(buf, cap, x.tobytes(), len(x), level)
    assert k <= cap
    return buf.raw[:k]


def both(frames, cap, skew=0):
    """(statuses, chunks) of the block-parallel and of the sequential decoder."""
    import torch
    lib = load()
    P = C.c_void_p
    lib.chucky_zstd_decode_chunks.argtypes = [P, P, P, C.c_size_t, P, C.c_size_t, C.c_size_t, P, P]
    n, stride = len(frames), cap + skew
    offs = np.cumsum([0] + [len(b) for b in frames[:-1]])
    blob = torch.from_numpy(np.frombuffer(b"".join(frames), np.uint8).copy()).cuda()
    d_off = torch.from_numpy(offs.astype("<i8")).cuda()
    d_len = torch.tensor([len(b) for b in frames], dtype=torch.int64, device="cuda")
    got = []
    for captured in (False, True):
        out = torch.full((n * stride + skew + 64,), 0xA5, dtype=torch.uint8, device="cuda")
        st = torch.full((n,), 99, dtype=torch.int32, device="cuda")

        def call():
            assert lib.chucky_zstd_decode_chunks(
                blob.data_ptr(), d_off.data_ptr(), d_len.data_ptr(), n, out.data_ptr() + skew,
                stride, cap, st.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0

        torch.cuda.synchronize()
        if captured:
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g):
                call()
            g.replay()
        else:
            call()
        torch.cuda.synchronize()
        raw = out.cpu().numpy()
        assert (raw[:skew] == 0xA5).all() and (raw[n * stride + skew:] == 0xA5).all()
        body = raw[skew:skew + n * stride].reshape(n, stride)
        assert (body[:, cap:] == 0xA5).all()  # nothing past a chunk
        got.append((st.cpu().numpy(), body[:, :cap]))
    return got


KINDS = ["poisson", "text", "rows", "runs", "mixed"]


@pytest.mark.parametrize("skew", [0, 1, 11])
@pytest.mark.parametrize("cap", [1, 100, 4096, 8191, 8193, 16384, 16385, 131072, 131073, 400001])
def test_stock_frames(cap, skew):
    x = [data(k, cap, cap + i) for i, k in enumerate(KINDS)]
    frames = [compress(v, level) for v in x for level in (-5, 1, 3, 9, 19)]
    for st, got in both(frames, cap, skew):
        assert (st == 0).all(), st
        for i, g in enumerate(got):
            assert np.array_equal(g, x[i // 5]), i


@pytest.mark.parametrize("cap", [2000, 16000, 140000])
def test_malformed_frames_keep_their_status(cap):
    rng = np.random.default_rng(cap)
    good = [compress(data(k, cap, i), lv) for i, k in enumerate(KINDS) for lv in (1, 12)]
    frames = []
    for g in good:
        frames += [g[:int(k)] for k in rng.integers(0, len(g), 6)] + [g + b"\0"]
        for k in rng.integers(0, min(len(g), 400), 8).tolist() + rng.integers(0, len(g), 8).tolist():
            b = bytearray(g)
            b[k] ^= int(rng.integers(1, 256))
            frames.append(bytes(b))
    frames.append(compress(data("text", cap // 2, 1), 3) + compress(data("rows", cap - cap // 2, 2), 3))
    frames.append((0x184D2A53).to_bytes(4, "little") + (5).to_bytes(4, "little") + b"hello" + good[0])
    frames.append(compress(data("text", cap - 1, 1), 3))
    frames.append(compress(data("text", cap + 1, 1), 3))
    (st, got), (want, ref) = both(frames, cap)
    assert np.array_equal(st, want)
    for i in np.flatnonzero(st == 0):
        assert np.array_equal(got[i], ref[i]), i
    assert st[-4] == 0 and st[-3] == 0 and st[-2] == 4 and st[-1] == 3


@pytest.mark.parametrize("level", [1, 3])
@pytest.mark.parametrize("cap", [3, 5000, 65536, 70001, 524288])
def test_own_frames(cap, level):
    import torch
    lib = load()
    lib.chucky_encode_bound.restype = lib.chucky_encode_scratch_bytes.restype = C.c_size_t
    P, Z = C.c_void_p, C.c_size_t
    lib.chucky_encode_bound.argtypes = [C.c_int, Z]
    lib.chucky_encode_scratch_bytes.argtypes = [C.c_int, C.c_int, Z, Z]
    lib.chucky_encode_chunks.argtypes = [C.c_int, C.c_int, P, Z, Z, Z, P, Z, P, P, Z, P]
    x = np.stack([data(k, cap, 7 + i) for i, k in enumerate(KINDS)])
    n, stride = len(x), (cap + 3) // 4 * 4
    buf = torch.zeros(n * stride + 256, dtype=torch.uint8, device="cuda")
    buf[:n * stride].view(n, stride)[:, :cap] = torch.from_numpy(x).cuda()
    ostride = lib.chucky_encode_bound(2, cap) + 16
    out = torch.zeros((n, ostride), dtype=torch.uint8, device="cuda")
    sizes = torch.zeros(n, dtype=torch.int64, device="cuda")
    sb = lib.chucky_encode_scratch_bytes(2, level, cap, n)
    scratch = torch.empty(sb, dtype=torch.uint8, device="cuda")
    assert lib.chucky_encode_chunks(2, level, buf.data_ptr(), cap, stride, n, out.data_ptr(), ostride,
                                    sizes.data_ptr(), scratch.data_ptr(), sb, None) == 0
    torch.cuda.synchronize()
    frames = [out[i, :k].cpu().numpy().tobytes() for i, k in enumerate(sizes.tolist())]
    for st, got in both(frames, cap, 3):
        assert (st == 0).all(), st
        assert np.array_equal(got, x)
