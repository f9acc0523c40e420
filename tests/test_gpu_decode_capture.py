"""A decoder call on one stream while another stream of the thread is being
captured, in every capture mode: the capture goes on and the chunks are
decoded, from the first call of a process on (which makes the scratch pool)."""
import subprocess
import sys

import pytest

import harness as H

pytestmark = pytest.mark.gpu

CODE = """
import ctypes as C
import sys
sys.path.insert(0, {root!r})
import torch
from chucky_gb300 import load
lib, P, Z = load(), C.c_void_p, C.c_size_t
call = lib.chucky_{codec}_decode_chunks
call.argtypes = [P, P, P, Z, P, Z, Z, P, P]
cap, n = 4096, 5
block = {block!r}
blob = torch.frombuffer(bytearray(block * n), dtype=torch.uint8).cuda()
lens = torch.full((n,), len(block), dtype=torch.int64, device="cuda")
offs = torch.arange(n, dtype=torch.int64, device="cuda") * len(block)
x = torch.zeros(8, device="cuda")
other = torch.cuda.Stream()
torch.cuda.synchronize()
for turn in range(2):
    out = torch.zeros(n * cap, dtype=torch.uint8, device="cuda")
    status = torch.full((n,), 99, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode={mode!r}):
        x.add_(1)
        assert call(blob.data_ptr(), offs.data_ptr(), lens.data_ptr(), n, out.data_ptr(), cap,
                    cap, status.data_ptr(), other.cuda_stream) == 0
        x.add_(1)
    torch.cuda.synchronize()
    assert status.tolist() == [0] * n
    assert (out == 65).all()
    g.replay()
    torch.cuda.synchronize()
    assert (x == 2 * (turn + 1)).all()
print("ok")
"""

# 4096 bytes 'A': an LZ4 block of one literal, a match of 4090 at offset 1 and
# five literals; a zstd frame (single segment, its size in 2 bytes) of one RLE
# block
BLOCKS = {
    "lz4": bytes([0x1F]) + b"A" + bytes([1, 0]) + bytes([255] * 15 + [4090 - 19 - 15 * 255])
           + bytes([0x50]) + b"A" * 5,
    "zstd": bytes([0x28, 0xB5, 0x2F, 0xFD, 0x60]) + (4096 - 256).to_bytes(2, "little")
            + (4096 << 3 | 1 << 1 | 1).to_bytes(3, "little") + b"A",
}


@pytest.mark.parametrize("mode", ["global", "thread_local", "relaxed"])
@pytest.mark.parametrize("codec", ["lz4", "zstd"])
def test_call_beside_a_capture(codec, mode):
    code = CODE.format(root=H.ROOT, codec=codec, block=BLOCKS[codec], mode=mode)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.endswith("ok\n")
