"""The zstd decoder's scratch: what the pool keeps is handed back by a call
without chunks, and a device with little room left decodes the blocks side by
side all the same, in smaller sets."""
import ctypes as C

import pytest
import torch

from chucky_gb300 import load
from test_gpu_zstd_decode_sets import encode

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def setup(cap, n):
    lib = load()
    P, Z = C.c_void_p, C.c_size_t
    lib.chucky_zstd_decode_chunks.argtypes = [P, P, P, Z, P, Z, Z, P, P]
    lib.chucky_launch_count.restype = C.c_uint64
    g = torch.Generator(device="cuda")
    g.manual_seed(cap)
    x = torch.randint(0, 9, (2, cap), generator=g, device="cuda", dtype=torch.uint8)
    f = encode(x, 1)
    blob = torch.cat(f)
    lens = torch.tensor([f[i % 2].numel() for i in range(n)], dtype=torch.int64, device="cuda")
    offs = torch.tensor([i % 2 * f[0].numel() for i in range(n)], dtype=torch.int64, device="cuda")
    out = torch.zeros((n, cap), dtype=torch.uint8, device="cuda")
    st = torch.full((n,), 99, dtype=torch.int32, device="cuda")

    def call(count=n):
        before = lib.chucky_launch_count()
        assert lib.chucky_zstd_decode_chunks(
            blob.data_ptr(), offs.data_ptr(), lens.data_ptr(), count, out.data_ptr(), cap, cap,
            st.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        return lib.chucky_launch_count() - before

    def check():
        assert (st == 0).all()
        for k in range(2):
            assert (out[k::2] == x[k]).all()
        st.fill_(99)
        out.zero_()

    return call, check


def free():
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def test_pool_is_handed_back():
    call, check = setup(MIB, 64)  # about 130 MiB of lists
    call(2)  # (the kernels are loaded at their first launch)
    call(0)
    before = free()
    assert call() == 6
    check()
    assert before - free() > 100 * MIB
    assert call(0) == 0
    assert before - free() < 16 * MIB


def test_little_room():
    call, check = setup(64 << 10, 4000)  # a set of 250 MiB
    call(2)
    call(0)
    room = free()
    hold = torch.empty(max(0, room - 60 * MIB), dtype=torch.uint8, device="cuda")
    try:
        launches = call()
    finally:
        del hold
        torch.cuda.empty_cache()
    check()
    # more than one set, and not the sequential kernel alone
    assert launches > 6
    call(0)
