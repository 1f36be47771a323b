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
    cdll.emu_index_records.restype = C.c_int64

    def check(text, words, mis=0, order=0):
        buf = as_u8(text)
        raw = np.full(-(-(buf.size + mis) // 16) * 16 + 32, 0x5B, np.uint8)  # brackets around it
        at = (-raw.ctypes.data) % 16 + mis
        raw[at:at + buf.size] = buf
        r = cdll.emu_arr_index(C.c_void_p(raw.ctypes.data + at), C.c_uint64(buf.size), words, order)
        assert r == 0, (r, cdll.emu_index_error(), words, mis, bytes(buf[:200]))

    check.lib = cdll
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


def record_starts(index, oracle, text, words, mis=0, order=0, cap=None):
    buf = as_u8(text)
    want = oracle.index(buf, 0 if words else 1)
    raw = np.full(-(-(buf.size + mis) // 16) * 16 + 32, 10 if words else 0x5B, np.uint8)
    at = (-raw.ctypes.data) % 16 + mis
    raw[at:at + buf.size] = buf
    got = np.full(max(want.size, 1) + 1, 0xEE, np.uint64)
    n = index.lib.emu_index_records(C.c_void_p(raw.ctypes.data + at), C.c_uint64(buf.size), words, C.c_void_p(got.ctypes.data), C.c_uint64(want.size if cap is None else cap), order)
    assert n == want.size, (n, want.size, index.lib.emu_index_error())
    keep = want.size if cap is None else min(cap, want.size)
    assert np.array_equal(got[:keep], want[:keep]) and (got[keep:] == 0xEE).all()


@pytest.mark.parametrize("words", [0, 1, 4])
def test_record_index(index, oracle, words):
    """k_nd_records and k_arr_records: separators on the edges of words and tiles, blank and empty lines, any alignment, too little room."""
    rng = random.Random(words)
    for it in range(12):
        flags = rng.choice([0, abi.PJ_GEN_ESCAPES, abi.PJ_GEN_WHITESPACE]) | (0 if words else abi.PJ_GEN_ARRAY)
        body = bytearray(pj.gen_text(4, it, 0, rng.choice([1, 50, 700]), flags))
        for _ in range(6):
            pos = rng.randrange(len(body) + 1)
            body[pos:pos] = rng.choice([b"\n", b"\n\n\n", b" \t\r\n", b"\n" + b" " * 70 + b"\n"] if words else [b",", b" ", b",,", b"[", b" ] "])
        record_starts(index, oracle, bytes(body), words, mis=it % 16, order=it, cap=None if it % 3 else 5)
    sep, fill = (b"\n", b"x") if words else (b",", b"1")
    for edge in (63, 64, 65, 16383, 16384, 16385, 65535, 65536, 65537):
        for mis in (0, 1, 15):
            body = fill * (edge - mis - 1) + sep + fill * 5 + sep + sep + b" " + sep + fill * 64
            record_starts(index, oracle, body if words else b"[" + body[1:] + b"]", words, mis)
    for body in (b"", sep, sep * 300, b" " * 70, b" " * 64 + sep, fill, b"[]", b"[ ]", b"[,]"):
        record_starts(index, oracle, body, words)
        record_starts(index, oracle, body, words, mis=15)


def test_lookbacks_on_states_of_tiles_side_by_side(index):
    """Many tiles back with nothing but their own functions or totals known, depths of all sizes, a tile that never comes."""
    rng = np.random.default_rng(8)
    n = 400
    st = rng.integers(0, 256, n).astype(np.uint8)
    d = rng.integers(-65536, 65537, (n, 4)).astype(np.int32)
    d[::7], d[3::11] = 65536, -65536
    agg = rng.integers(0, 1 << 40, n).astype(np.uint64)
    back = lambda tile, known, missing=n: (
        index.lib.emu_arr_lookback(n, tile, C.c_void_p(st.ctypes.data), C.c_void_p(d.ctypes.data), known, tile % 4, [0, -70000, 1 << 30, 5][tile % 4], missing),
        index.lib.emu_sum_lookback(n, tile, C.c_void_p(agg.ctypes.data), known, C.c_uint64(1 << 45), missing))
    for tile in (1, 2, 31, 32, 33, 64, 65, 127, 128, 129, 161, 256, 257, 399):
        for known in sorted({-1, 0, tile // 2, max(tile - 129, -1), max(tile - 33, -1), max(tile - 32, -1), max(tile - 31, -1), tile - 2, tile - 1}):
            if known < tile:
                assert back(tile, known) == (0, 0), (tile, known)
        assert back(tile, -1, missing=0) == (2, 2)  # (the totals of the others do not help)
        if tile > 40:
            assert back(tile, tile - 5, missing=tile - 20) == (0, 0)  # nobody needs that one


@pytest.mark.skipif(os.environ.get("PJ_EMU_SANITIZE") == "1", reason="is the run under the sanitizers")
def test_under_sanitizers():
    asan = subprocess.run(["gcc", "-print-file-name=libasan.so"], capture_output=True, text=True).stdout.strip()
    env = dict(os.environ, PJ_EMU_SANITIZE="1", LD_PRELOAD=asan, ASAN_OPTIONS="detect_leaks=0:detect_stack_use_after_return=0")
    r = subprocess.run([sys.executable, "-m", "pytest", "-q", "-x", "-p", "no:cacheprovider", __file__, "-k", "mutated or runs and 65 or record_index and 4"], env=env, capture_output=True, text=True, cwd=ROOT)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-3000:]
