"""k_arr_index (csrc/pj_array_index.cuh) run on the CPU, block by block, against the same rules word after word: no GPU needed."""
import ctypes as C
import os
import random
import subprocess
import sys

import numpy as np
import pytest

from pj_testlib import abi, as_u8, pj

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="session")
def index():
    src = os.path.join(HERE, "host_emu", "pj_index_emu.cpp")
    csrc = os.path.join(ROOT, "micronaut3-bug_b200", "csrc")
    deps = [src, os.path.join(HERE, "host_emu", "pj_block_emu.h")] + [os.path.join(csrc, f) for f in os.listdir(csrc) if f.endswith((".cuh", ".h", ".inc"))]
    san = os.environ.get("PJ_EMU_SANITIZE") == "1"
    flags = ["-O1", "-g", "-fsanitize=address,undefined", "-fno-sanitize-recover=all"] if san else ["-O2"]
    lib = os.path.join(HERE, "host_emu", f"libpj_index_emu{'_san' if san else ''}.so")
    if not os.path.exists(lib) or any(os.path.getmtime(d) > os.path.getmtime(lib) for d in deps):
        subprocess.run(["g++", *flags, "-std=c++17", "-fno-extern-tls-init", "-fPIC", "-shared", "-w", "-I", os.path.join(ROOT, "include"), "-I", csrc, "-x", "c++", src, "-o", lib], check=True)
    cdll = C.CDLL(lib)
    cdll.emu_index_error.restype = C.c_char_p

    def check(text, words, mis=0, order=0):
        buf = as_u8(text)
        raw = np.full(-(-(buf.size + mis) // 16) * 16 + 32, 0x5B, np.uint8)  # brackets around it
        at = (-raw.ctypes.data) % 16 + mis
        raw[at:at + buf.size] = buf
        r = cdll.emu_arr_index(C.c_void_p(raw.ctypes.data + at), C.c_uint64(buf.size), words, order)
        assert r == 0, (r, cdll.emu_index_error(), words, mis, bytes(buf[:200]))

    return check


SPECIAL = [b'"', b"\\", b"\\\\", b'\\"', b"[", b"]", b"{", b"}", b",", b" ", b"\n", b"\\" * 63, b"\\" * 64, b"\\" * 65, b'"a,b]"', b"[]", b"x", b"\xc3\xa9", b"}" * 70, b"|;=\xfb\xfd\xdb\xdd"]


@pytest.mark.parametrize("words", [1, 4])
def test_mutated_arrays(index, words):
    rng = random.Random(words)
    for it in range(40):
        flags = abi.PJ_GEN_ARRAY | rng.choice([0, abi.PJ_GEN_ESCAPES, abi.PJ_GEN_WHITESPACE, abi.PJ_GEN_ESCAPES | abi.PJ_GEN_MALFORMED])
        body = bytearray(pj.gen_text(rng.choice([1, 4]), it, 0, rng.choice([1, 30, 300]), flags))
        for _ in range(rng.randrange(0, 8)):
            pos = rng.randrange(len(body) + 1)
            body[pos:pos] = rng.choice(SPECIAL)
        if it % 5 == 0:
            body = body[: rng.randrange(len(body))]
        index(bytes(body), words, mis=rng.choice([0, 0, 1, 7, 8, 15]), order=it % 7)


@pytest.mark.parametrize("run", [1, 63, 64, 65, 127, 128, 255, 256, 257, 16383, 16384, 16385, 65536])
def test_backslash_runs(index, run):
    """Escape parity, in-string state and depth carry across words, threads and tiles."""
    for lead in (0, 1, 17, 250):
        body = b"[" + b" " * lead + b'{"name":"' + b"\\" * run + b'","photoUrls":["[,]{}"]},{"name":"b","photoUrls":[]}]'
        for words in (1, 4):
            index(body, words, mis=lead % 16)


@pytest.mark.parametrize("words", [1, 4])
def test_shapes(index, words):
    index(b"", words)
    for text in (b"[", b"]", b"[]", b" [ ] ", b'[1,"a,]",{},[2,[3]],,] [4]', b"{", b'"[', b"]]][[["):
        for mis in (0, 15):
            index(text, words, mis)
    index(b"[" + b"1," * 40000 + b"2]", words, 3)  # every word full of separators
    index(b"[" * 70000 + b"]" * 70000, words)  # depths as large as a tile
    index(b"]" * 40000 + b"[" * 40001, words, 9)
    index(b'["' + b"x" * 140000 + b'",1]', words)


@pytest.mark.skipif(os.environ.get("PJ_EMU_SANITIZE") == "1", reason="is the run under the sanitizers")
def test_under_sanitizers():
    asan = subprocess.run(["gcc", "-print-file-name=libasan.so"], capture_output=True, text=True).stdout.strip()
    env = dict(os.environ, PJ_EMU_SANITIZE="1", LD_PRELOAD=asan, ASAN_OPTIONS="detect_leaks=0:detect_stack_use_after_return=0")
    r = subprocess.run([sys.executable, "-m", "pytest", "-q", "-x", "-p", "no:cacheprovider", __file__, "-k", "mutated or runs and 65"], env=env, capture_output=True, text=True, cwd=ROOT)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-3000:]
