"""Calls of the zstd decoder so large that its lists are filled more than once,
and that one warp decodes several blocks, a lane each: this library's frames of
512 KiB and 1 MiB chunks, levels 1 and 3, with frames behind the first set that
the block-parallel decoder leaves (a skippable frame in front, two frames, a
byte cut off or added)."""
import ctypes as C

import numpy as np
import pytest
import torch

from chucky_gb300 import load
from test_gpu_zstd_decode_blocks import compress

pytestmark = pytest.mark.gpu

KIB = 1 << 10


def encode(x, level):
    """x: [n, cap] device bytes -> their frames, a list of device tensors."""
    lib = load()
    P, Z = C.c_void_p, C.c_size_t
    lib.chucky_encode_bound.restype = lib.chucky_encode_scratch_bytes.restype = Z
    lib.chucky_encode_bound.argtypes = [C.c_int, Z]
    lib.chucky_encode_scratch_bytes.argtypes = [C.c_int, C.c_int, Z, Z]
    lib.chucky_encode_chunks.argtypes = [C.c_int, C.c_int, P, Z, Z, Z, P, Z, P, P, Z, P]
    n, cap = x.shape
    stride = lib.chucky_encode_bound(2, cap) // 16 * 16 + 16
    buf = torch.cat([x.reshape(-1), x.new_zeros(256)])
    out = x.new_zeros((n, stride))
    sizes = torch.zeros(n, dtype=torch.int64, device="cuda")
    sb = lib.chucky_encode_scratch_bytes(2, level, cap, n)
    scratch = torch.empty(sb, dtype=torch.uint8, device="cuda")
    assert lib.chucky_encode_chunks(2, level, buf.data_ptr(), cap, cap, n, out.data_ptr(), stride,
                                    sizes.data_ptr(), scratch.data_ptr(), sb, None) == 0
    return [out[i, :k] for i, k in enumerate(sizes.tolist())]


@pytest.mark.parametrize("cap,n,level", [(512 * KIB, 64, 1), (512 * KIB, 64, 3),
                                         (512 * KIB, 600, 3), (1024 * KIB, 300, 1)])
def test_large_calls(cap, n, level):
    g = torch.Generator(device="cuda")
    g.manual_seed(n + level)
    kinds = 16
    x = torch.randint(0, 16, (kinds, cap), generator=g, device="cuda", dtype=torch.uint8)
    e = torch.arange(cap, device="cuda")
    for i in range(0, kinds, 4):
        x[i] += ((e // 2 % 64) ^ (e // 128 % 64) ^ (e // 8192 + i)).to(torch.uint8)  # texture
        x[i + 1] = x[i, :3000].repeat(cap // 3000 + 1)[:cap]                         # long matches
        x[i + 2] = i                                                                 # constant
    frames = encode(x, level)
    skip = torch.tensor([0x53, 0x2A, 0x4D, 0x18, 2, 0, 0, 0, 9, 9], dtype=torch.uint8, device="cuda")
    half = np.frombuffer(compress(np.full(cap // 2, 6, np.uint8), 1), np.uint8).copy()
    two = torch.from_numpy(np.concatenate([half, half])).cuda()
    f, want, status = [], [], []
    for i in range(n):
        k = (5 * i + i // kinds) % kinds
        b, w, s = frames[k], x[k], 0
        if i % 37 == 36:
            b, w, s = [(torch.cat([skip, frames[2]]), x[2], 0), (two, x.new_full((cap,), 6), 0),
                       (frames[2][:-1], x[2], 1),
                       (torch.cat([frames[2], skip[-1:]]), x[2], 1)][i // 37 % 4]
        f.append(b)
        want.append(w)
        status.append(s)
    blob = torch.cat(f)
    lens = torch.tensor([b.numel() for b in f], dtype=torch.int64, device="cuda")
    offs = torch.cumsum(lens, 0) - lens
    out = torch.full((n, cap), 0xA5, dtype=torch.uint8, device="cuda")
    st = torch.full((n,), 99, dtype=torch.int32, device="cuda")
    lib = load()
    P, Z = C.c_void_p, C.c_size_t
    lib.chucky_zstd_decode_chunks.argtypes = [P, P, P, Z, P, Z, Z, P, P]
    assert lib.chucky_zstd_decode_chunks(blob.data_ptr(), offs.data_ptr(), lens.data_ptr(), n,
                                         out.data_ptr(), cap, cap, st.data_ptr(),
                                         torch.cuda.current_stream().cuda_stream) == 0
    got = st.tolist()
    assert [min(s, 1) for s in got] == status, got
    for i in range(n):
        if status[i] == 0:
            assert torch.equal(out[i], want[i]), i
