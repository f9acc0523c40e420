"""The LZ4 decoder on more blocks than the chip holds CTAs for, where a CTA
takes several blocks and a warp of it tries each first: blocks that a warp
keeps, leaves at once, or leaves after some sequences (dense, sparse, one
literal run, constant, sparse before dense and the other way round), cut short
or with a byte changed, around the sizes and counts where the form changes.
Statuses and bytes must be the sequential decoder's."""
import numpy as np
import pytest
import torch

import test_gpu_lz4_decode_tiles as T

pytestmark = pytest.mark.gpu


def sequences(parts, cap, seed):
    """A block of `cap` bytes: `parts` lists (output bytes, literal lengths,
    match lengths, offsets) to draw sequences from, one after the other."""
    rng = np.random.default_rng(seed)
    block, out = bytearray(), 0
    for upto, lits, matches, offs in parts:
        while out < upto:
            lit, ml = int(rng.choice(lits)), int(rng.choice(matches))
            lit += out == 0 and lit == 0
            if out + lit + ml + 5 > cap:
                break
            off = min(out + lit, int(rng.choice(offs)))
            block += bytes([min(lit, 15) << 4 | min(ml - 4, 15)])
            block += T._len(lit) if lit >= 15 else b""
            block += rng.integers(0, 256, lit, dtype=np.uint8).tobytes()
            block += bytes([off & 255, off >> 8])
            block += T._len(ml - 4) if ml - 4 >= 15 else b""
            out += lit + ml
    lit = cap - out
    block += bytes([min(lit, 15) << 4]) + (T._len(lit) if lit >= 15 else b"")
    return bytes(block + rng.integers(0, 256, lit, dtype=np.uint8).tobytes())


DENSE = ([0, 1, 3, 5, 9], [4, 5, 6, 20], [1, 2, 3, 8, 100, 5000])
SPARSE = ([80, 200, 400, 700], [4, 5], [40, 1000, 60000])
CONSTANT = ([0, 1], [600, 1500, 2500], [1, 2])
LONG = ([524, 525, 1023, 1024, 2054, 2055, 4000], [4, 528, 529, 1024, 2058, 2059], [1, 7, 300])


def kinds(cap, seed):
    half = cap // 2
    b = [sequences([(cap,) + DENSE], cap, seed), sequences([(cap,) + SPARSE], cap, seed + 1),
         sequences([(cap,) + CONSTANT], cap, seed + 2), sequences([], cap, seed + 3),
         sequences([(half,) + SPARSE, (cap,) + DENSE], cap, seed + 4),
         sequences([(half,) + DENSE, (cap,) + CONSTANT], cap, seed + 5),
         sequences([(cap,) + LONG], cap, seed + 6)]
    rng = np.random.default_rng(seed)
    for g in list(b):
        b.append(g[:int(rng.integers(0, len(g)))])
        c = bytearray(g)
        c[int(rng.integers(0, len(g)))] ^= int(rng.integers(1, 256))
        b.append(bytes(c))
        b.append(g + b"\0")
    return b


def count(per_sm):
    return per_sm * torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("skew", [0, 5])
@pytest.mark.parametrize("cap", [7, 256, 257, 1024, 1025, 4096, 4440, 9000, 40000])
@pytest.mark.parametrize("per_sm", [8, 12, 16, 33])
def test_many_blocks(per_sm, cap, skew):
    n = count(per_sm) + 1
    if n * cap > 64 << 20:
        n = count(8) + 1
    k = kinds(cap, cap)
    blocks = [k[(i + i // len(k)) % len(k)] for i in range(n)]
    st, got = T.run(blocks, cap, skew)
    known = {b: T.decode(b, cap) for b in set(k)}
    assert (st == [known[b][0] for b in blocks]).all()
    for b in set(k):
        if known[b][0] == 0:
            want = np.frombuffer(bytes(known[b][1]), np.uint8)
            rows = got[[i for i, x in enumerate(blocks) if x == b]]
            assert (rows == want).all()


@pytest.mark.parametrize("cap", [16384, 16385, 70000])
@pytest.mark.parametrize("per_sm", [1, 2])
def test_large_blocks(per_sm, cap):
    """Where the large CTAs give way to small ones, and long sequences are
    copied without a window."""
    k = kinds(cap, 3 * cap)
    for n in (count(per_sm), count(per_sm) + 1):
        T.check([k[i % len(k)] for i in range(n)], cap)
