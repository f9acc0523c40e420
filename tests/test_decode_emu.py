"""The decoders' forms for large calls, reached with few chunks: the CPU
emulation of the kernels (AddressSanitizer and UBSan where the compiler has
them) built for a chip that holds one small LZ4 CTA, so that a CTA takes
several blocks and its warps try them first."""
import os
import shutil
import subprocess

import pytest

import harness as H

EMU = os.path.join(H.ROOT, "tests", "emu")
OUT = os.path.join(EMU, "_build", "decode_emu")
LARGE = ["-DCHUCKY_LZ4_SLOTS(sms)=1"]

# blocks of few sequences, of many, of one, constant ones, and one after the
# other in a chunk; a block left at its start, after some sequences, never;
# CTAs with a block to spare
CASES = [("lz4", p, c, n) for p in ("mixed", "random", "xor16", "geom", "halves", "zeros")
         for c, n in ((3000, 5), (9000, 4))]
CASES += [("lz4", "geom", 700, 7), ("lz4", "mixed", 700, 8), ("lz4", "xor16", 200, 3),
          ("lz4", "ramp", 5000, 3)]


@pytest.fixture(scope="module")
def emu():
    if not shutil.which("g++"):
        pytest.skip("g++ not available")
    if not (H.oracle().oracle_codecs_available() & 3) == 3:
        pytest.skip("stock liblz4/libzstd not available")
    os.makedirs(os.path.dirname(OUT), exist_ok=True)
    base = ["g++", "-std=c++20", "-O1", "-g", *LARGE, "-I", os.path.join(EMU, "fake"),
            "-I", os.path.join(H.ROOT, "include"),
            "-I", os.path.join(H.ROOT, "chucky_gb300", "csrc"),
            os.path.join(EMU, "codec_emu.cpp"), os.path.join(EMU, "simt.cpp"),
            "-o", OUT, "-ldl", "-lpthread"]
    san = ["-fsanitize=address,undefined", "-fno-sanitize-recover=all"]
    r = subprocess.run(base[:1] + san + base[1:], capture_output=True, text=True)
    if r.returncode != 0:  # no sanitizer runtime: plain build
        r = subprocess.run(base, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return OUT


@pytest.mark.parametrize("codec,pattern,chunk,n", CASES)
def test_large_call_forms(emu, codec, pattern, chunk, n):
    r = subprocess.run([emu, codec, str(chunk), str(n), pattern, "11"], capture_output=True,
                       text=True, timeout=900)
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.startswith("ok")
