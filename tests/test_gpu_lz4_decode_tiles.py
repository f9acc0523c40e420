"""The tiled LZ4 decoder against a plain sequential decoder (below) on blocks
made sequence by sequence: lengths around the token's 15, the 255 of a length
byte and the longest a window follows, offsets of 1 up to the whole chunk
(overlapping, into the tile, before it), chunks around one and several tiles,
both thread counts, every input and output alignment; and the same blocks cut
short or with a byte changed, whose statuses must be the sequential ones."""
import ctypes as C

import numpy as np
import pytest

from chucky_gb300 import load

pytestmark = pytest.mark.gpu


def decode(block, cap):
    """(status, bytes) as include/chucky_gb300.h declares them."""
    ip, out, n = 0, bytearray(), len(block)

    def length(v):
        nonlocal ip
        while v >= 15:
            if ip >= n:
                return None
            ip += 1
            v += block[ip - 1]
            if block[ip - 1] != 255:
                break
        return v

    while True:
        if ip >= n:
            return 1, out
        tok = block[ip]
        ip += 1
        lit = length(tok >> 4)
        if lit is None or lit > n - ip:
            return 1, out
        if lit > cap - len(out):
            return 3, out
        out += block[ip:ip + lit]
        ip += lit
        if ip == n:
            return (0 if len(out) == cap else 4), out
        if n - ip < 2:
            return 1, out
        off = block[ip] | block[ip + 1] << 8
        ip += 2
        if off == 0 or off > len(out):
            return 2, out
        ml = length(tok & 15)
        if ml is None:
            return 1, out
        ml += 4
        if ml > cap - len(out):
            return 3, out
        for k in range(0, ml, off):
            out += out[-off:][:ml - k] if off <= ml - k else out[len(out) - off:][:ml - k]


def _len(v):
    b = bytearray()
    v -= 15
    while v >= 255:
        b.append(255)
        v -= 255
    b.append(v)
    return b


def make_block(cap, seed, long_lengths):
    """A valid block of `cap` output bytes."""
    rng = np.random.default_rng(seed)
    block, out = bytearray(), 0
    lens = [0, 1, 3, 14, 15, 16, 40, 269, 270, 271] + (
        [4000, 8170, 8174, 8175, 8176, 17000, 70000] if long_lengths else [])
    p = np.ones(len(lens))
    p[:6] = 30
    p /= p.sum()
    while True:
        lit = int(rng.choice(lens, p=p))
        ml = 4 + int(rng.choice(lens, p=p))
        if out == 0 and lit == 0:
            lit = 1
        if out + lit + ml + 5 > cap:
            lit = cap - out
            block += bytes([min(lit, 15) << 4]) + (_len(lit) if lit >= 15 else b"")
            block += rng.integers(0, 256, lit, dtype=np.uint8).tobytes()
            return bytes(block)
        have = out + lit
        off = int(min(have, 65535, rng.choice([1, 2, 3, 4, 7, 16, 100, 5000, 65535])))
        block += bytes([min(lit, 15) << 4 | min(ml - 4, 15)])
        block += _len(lit) if lit >= 15 else b""
        block += rng.integers(0, 256, lit, dtype=np.uint8).tobytes()
        block += bytes([off & 255, off >> 8])
        block += _len(ml - 4) if ml - 4 >= 15 else b""
        out += lit + ml


def run(blocks, cap, skew=0):
    import torch
    lib = load()
    P = C.c_void_p
    lib.chucky_lz4_decode_chunks.argtypes = [P, P, P, C.c_size_t, P, C.c_size_t, C.c_size_t, P, P]
    n, stride = len(blocks), cap + skew
    offs = np.cumsum([0] + [len(b) for b in blocks[:-1]])
    blob = torch.from_numpy(np.frombuffer(b"".join(blocks) or b"\0", np.uint8).copy()).cuda()
    d_off = torch.from_numpy(offs.astype("<i8")).cuda()
    d_len = torch.tensor([len(b) for b in blocks], dtype=torch.int64, device="cuda")
    out = torch.full((n * stride + skew + 64,), 0xA5, dtype=torch.uint8, device="cuda")
    st = torch.full((n,), 99, dtype=torch.int32, device="cuda")
    assert lib.chucky_lz4_decode_chunks(blob.data_ptr(), d_off.data_ptr(), d_len.data_ptr(), n,
                                        out.data_ptr() + skew, stride, cap, st.data_ptr(), None) == 0
    torch.cuda.synchronize()
    raw = out.cpu().numpy()
    assert (raw[:skew] == 0xA5).all() and (raw[n * stride + skew:] == 0xA5).all()
    got = raw[skew:skew + n * stride].reshape(n, stride)
    assert (got[:, cap:] == 0xA5).all()  # nothing past a chunk
    return st.cpu().numpy(), got[:, :cap]


@pytest.mark.parametrize("skew", [0, 1, 13])
@pytest.mark.parametrize("cap", [1, 5, 4095, 4096, 4097, 16384, 16385, 32768, 50001, 300000])
@pytest.mark.parametrize("long_lengths", [False, True])
def test_valid_blocks(cap, long_lengths, skew):
    blocks = [make_block(cap, 100 * cap + s, long_lengths) for s in range(6)]
    st, got = run(blocks, cap, skew)
    for b, s, g in zip(blocks, st, got):
        want, data = decode(b, cap)
        assert want == 0 and s == 0
        assert g.tobytes() == bytes(data)


@pytest.mark.parametrize("cap", [300, 5000, 40000])
def test_malformed_blocks_keep_their_status(cap):
    rng = np.random.default_rng(cap)
    blocks = []
    for s in range(8):
        b = make_block(cap, s, s % 2 == 1)
        blocks += [b[:int(k)] for k in rng.integers(0, len(b), 12)]
        for k in rng.integers(0, len(b), 12):
            c = bytearray(b)
            c[int(k)] = int(rng.integers(0, 256))
            blocks.append(bytes(c))
        blocks.append(b + b"\0")
    st, got = run(blocks, cap)
    for b, s, g in zip(blocks, st, got):
        want, data = decode(b, cap)
        assert s == want
        if want == 0:
            assert g.tobytes() == bytes(data)


def check(blocks, cap):
    st, got = run(blocks, cap)
    known = {b: decode(b, cap) for b in set(blocks)}
    for b, s, g in zip(blocks, st, got):
        want, data = known[b]
        assert s == want
        if want == 0:
            assert g.tobytes() == bytes(data)


@pytest.mark.parametrize("cap", [4097, 16384, 16385, 60000])
@pytest.mark.parametrize("n", [1, 2, 76, 77, 152, 153, 457])
def test_block_counts(n, cap):
    """Two CTAs to a block, one large one, or one small one."""
    kinds = [make_block(cap, s, s % 2 == 1) for s in range(5)]
    check([kinds[i % 5] for i in range(n)], cap)


@pytest.mark.parametrize("seed", range(6))
def test_few_malformed_blocks(seed):
    """... of which some break off, and others are whole."""
    cap, rng = 40000, np.random.default_rng(1000 + seed)
    blocks = []
    for s in range(8):
        b = bytearray(make_block(cap, 10 * seed + s, s % 2 == 1))
        if s % 4 == 1:
            del b[int(rng.integers(0, len(b))):]
        elif s % 4:
            b[int(rng.integers(0, len(b)))] = int(rng.integers(0, 256))
        blocks.append(bytes(b))
    check(blocks, cap)
