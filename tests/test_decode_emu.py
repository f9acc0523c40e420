"""The decoders' forms for large calls, reached with few chunks: the CPU
emulation of the kernels (AddressSanitizer and UBSan where the compiler has
them) built for a chip that holds one small LZ4 CTA, so that a CTA takes
several blocks and its warps try them first, and with little room for the zstd
decoder's lists, so that a call takes several launch sets."""
import os
import shutil
import subprocess

import pytest

import harness as H

EMU = os.path.join(H.ROOT, "tests", "emu")
BUILD = os.path.join(EMU, "_build")

# blocks of few sequences, of many, of one, constant ones, and one after the
# other in a chunk; a block left at its start, after some sequences, never;
# CTAs with a block to spare
CASES = [("lz4", p, c, n) for p in ("mixed", "random", "xor16", "geom", "halves", "zeros")
         for c, n in ((3000, 5), (9000, 4))]
CASES += [("lz4", "geom", 700, 7), ("lz4", "mixed", 700, 8), ("lz4", "xor16", 200, 3),
          ("lz4", "ramp", 5000, 3)]



def build(source, name, *flags):
    if not shutil.which("g++"):
        pytest.skip("g++ not available")
    if not (H.oracle().oracle_codecs_available() & 3) == 3:
        pytest.skip("stock liblz4/libzstd not available")
    os.makedirs(BUILD, exist_ok=True)
    out = os.path.join(BUILD, name)
    base = ["g++", "-std=c++20", "-O1", "-g", *flags, "-I", os.path.join(EMU, "fake"),
            "-I", os.path.join(H.ROOT, "include"),
            "-I", os.path.join(H.ROOT, "chucky_gb300", "csrc"),
            os.path.join(EMU, source), os.path.join(EMU, "simt.cpp"),
            "-o", out, "-ldl", "-lpthread"]
    san = ["-fsanitize=address,undefined", "-fno-sanitize-recover=all"]
    r = subprocess.run(base[:1] + san + base[1:], capture_output=True, text=True)
    if r.returncode != 0:  # no sanitizer runtime: plain build
        r = subprocess.run(base, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return out


def run(*cmd):
    r = subprocess.run([str(c) for c in cmd], capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.startswith("ok")
    return r.stdout


@pytest.fixture(scope="module")
def emu():
    return build("codec_emu.cpp", "codec_emu_large", "-DCHUCKY_LZ4_SLOTS(sms)=1")


@pytest.mark.parametrize("codec,pattern,chunk,n", CASES)
def test_large_call_forms(emu, codec, pattern, chunk, n):
    run(emu, codec, chunk, n, pattern, 11)


@pytest.fixture(scope="module")
def decode_emu():
    return build("decode_emu.cpp", "decode_emu", "-DCHUCKY_ZSTD_SCRATCH=40000",
                 "-DCHUCKY_ZSTD_FRAMES=10")


@pytest.mark.parametrize("chunk,per_set", [(3000, 4), (1200, 8), (30000, 1)])
@pytest.mark.parametrize("n", [1, 9, 10, 23])
def test_launch_sets(decode_emu, chunk, per_set, n):
    """Chunks past the first launch set, the last one of any size; the
    sequential decoder runs once over all the chunks whose records are kept
    (ten here), not once per set."""
    per_set = min(per_set, n)
    groups = [min(10, n - g) for g in range(0, n, 10)]
    want = sum(5 * -(-g // per_set) + 1 for g in groups)
    assert run(decode_emu, chunk, n, 3 * chunk + n) == "ok %d\n" % want


@pytest.mark.parametrize("chunk,launches", [(64, 1), (65, 6)])
def test_tiny_chunks(decode_emu, chunk, launches):
    """Chunks up to 64 bytes go to the sequential decoder at once."""
    assert run(decode_emu, chunk, 8, chunk) == "ok %d\n" % launches
