"""k_write_tile (csrc/pj_write_tile.cuh) run on the CPU, block by block, against the checker: no GPU needed (tests/host_emu/pj_block_emu.h)."""
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
NDJSON, ARRAY = abi.PJ_FRAMING_NDJSON, abi.PJ_FRAMING_ARRAY
PET, ORDER, USER, MIXED = abi.PJ_SCHEMA_PET, abi.PJ_SCHEMA_ORDER, abi.PJ_SCHEMA_USER, abi.PJ_SCHEMA_MIXED
INCLUSIONS = [abi.PJ_INCLUDE_NON_EMPTY, abi.PJ_INCLUDE_NON_NULL, abi.PJ_INCLUDE_ALWAYS]
COL = {c.name: c.id for c in abi.schema_columns(MIXED)}
ESC, SPARSE, BAD, ZIPF = abi.PJ_GEN_ESCAPES, abi.PJ_GEN_SPARSE, abi.PJ_GEN_MALFORMED, abi.PJ_GEN_ZIPF_LISTS


@pytest.fixture(scope="session")
def writer():
    src = os.path.join(HERE, "host_emu", "pj_write_emu.cpp")
    csrc = os.path.join(ROOT, "micronaut3-bug_b200", "csrc")
    deps = [src, os.path.join(HERE, "host_emu", "pj_block_emu.h")] + [os.path.join(csrc, f) for f in os.listdir(csrc) if f.endswith((".cuh", ".h", ".inc"))]
    san = os.environ.get("PJ_EMU_SANITIZE") == "1"
    flags = ["-O1", "-g", "-fsanitize=address,undefined", "-fno-sanitize-recover=all"] if san else ["-O2"]
    lib = os.path.join(HERE, "host_emu", f"libpj_write_emu{'_san' if san else ''}.so")
    if not os.path.exists(lib) or any(os.path.getmtime(d) > os.path.getmtime(lib) for d in deps):
        subprocess.run(["g++", *flags, "-std=c++17", "-fno-extern-tls-init", "-fPIC", "-shared", "-w", "-I", os.path.join(ROOT, "include"), "-I", csrc, "-x", "c++", src, "-o", lib], check=True)
    cdll = C.CDLL(lib)
    cdll.emu_write_error.restype = C.c_char_p
    return cdll


def write(lib, schema, cols, want, framing=NDJSON, inclusion=abi.PJ_INCLUDE_NON_NULL, recs=128, shared=65536, mis=0, order=0, lower=0):
    """Compares the emulated kernel's text with `want`; array framing: without the brackets, which another kernel writes."""
    text = want[1:-1] if framing == ARRAY else want
    raw = np.full(text.size + 96, 0xEE, np.uint8)
    at = (-raw.ctypes.data) % 16 + 16 + mis
    n = C.c_uint64()
    out = C.c_void_p(raw.ctypes.data + at - (1 if framing == ARRAY else 0))
    st = lib.emu_write_tiles(schema, int(framing == ARRAY), inclusion, lower, C.byref(cols.raw), out, C.c_uint64(text.size + 2), recs, shared, order, C.byref(n))
    assert st >= 0, lib.emu_write_error().decode()
    got = raw[at:at + text.size]
    size = int(n.value) - (1 if framing == ARRAY and n.value else 0)
    assert st == 0 and size == text.size, (size, text.size)
    if not np.array_equal(got, text):
        k = int(np.argmax(got != text))
        raise AssertionError((k, bytes(got[max(0, k - 40):k + 40]), bytes(text[max(0, k - 40):k + 40])))
    behind = raw[at + text.size + (1 if framing == ARRAY and n.value else 0):]
    assert (raw[:at] == 0xEE).all() and (behind == 0xEE).all()


SHAPES = [dict(), dict(recs=32, shared=24576, mis=5), dict(recs=256, shared=131072, mis=15, order=3), dict(recs=96, shared=40960, mis=8, order=6), dict(recs=5, shared=8192, mis=1)]


@pytest.mark.parametrize("schema", [PET, ORDER, USER, MIXED])
@pytest.mark.parametrize("flags", [0, ESC, SPARSE, ESC | SPARSE | BAD, ZIPF | ESC])
def test_generated_tables(writer, oracle, schema, flags):
    n = 60 if flags & ZIPF else 300
    cols = oracle.parse(schema, pj.gen_text(schema, 0xE12, 0, n, flags))
    for k, shape in enumerate(SHAPES):
        for framing in (NDJSON, ARRAY):
            for inclusion in INCLUSIONS if k < 2 else INCLUSIONS[1:2]:
                write(writer, schema, cols, oracle.write(schema, cols, framing, inclusion), framing, inclusion, **shape)


def edge_text(rng, n):
    """Pets with strings of every length around the words, bytes to escape of every kind, long and empty lists, integers of every length."""
    def s():
        k = rng.choice([0, 1, 2, 3, 4, 5, 7, 8, 9, 15, 16, 17, 31, 33, 64, 600])
        return "".join(rng.choice(['a', 'b', '\\"', "\\\\", "\\n", "\\u0001", "\\u001f", "é", "/"] if rng.random() < 0.3 else ["x"]) for _ in range(k))

    def i():
        return str(rng.choice([0, 1, -1, 9, 10, 99999999, 100000000, 9999999999999999, 10000000000000000, -9223372036854775808, 9223372036854775807,
                               rng.randrange(10 ** rng.randrange(1, 19)), -rng.randrange(10 ** rng.randrange(1, 19))]))
    out = []
    for _ in range(n):
        tags = ",".join(rng.choice(["{}", '{"id":%s}' % i(), '{"name":"%s"}' % s(), '{"id":%s,"name":"%s"}' % (i(), s())]) for _ in range(rng.choice([0, 1, 2, 3, 40])))
        urls = ",".join('"%s"' % s() for _ in range(rng.choice([0, 0, 1, 2, 5, 33])))
        p = ['"id":%s' % i(), rng.choice(['"category":{}', '"category":{"id":%s,"name":"%s"}' % (i(), s()), '"category":null']), '"name":"%s"' % s(), '"photoUrls":[%s]' % urls,
             '"tags":[%s]' % tags, '"status":"%s"' % rng.choice(["available", "pending", "sold"])]
        out.append("{" + ",".join(x for k, x in enumerate(p) if k in (2, 3) or rng.random() < 0.7) + "}")
    return as_u8("\n".join(out).encode())


@pytest.mark.parametrize("seed", range(6))
def test_edges(writer, oracle, seed):
    """Rounds of a window too small for the tile, more strings with escapes than a round keeps, records larger than the window."""
    rng = random.Random(seed)
    cols = oracle.parse(PET, edge_text(rng, 90))
    assert cols.n_errors == 0
    for shape in [dict(recs=32, shared=65536), dict(recs=8, shared=16384, mis=7), dict(recs=128, shared=128 * 1024, mis=3, order=5), dict(recs=1, shared=8192, mis=9), dict(recs=16, shared=12288, mis=2)]:
        for inclusion in INCLUSIONS:
            write(writer, PET, cols, oracle.write(PET, cols, NDJSON, inclusion), inclusion=inclusion, **shape)


def test_dates(writer, oracle):
    rng = random.Random(4)
    lines = []
    for y in (0, 1, 99, 100, 1582, 1969, 1970, 1999, 2000, 2024, 2100, 9999):
        for frac in ("", ".5", ".000000001", ".123456789", ".120", ".00001"):
            for off in ("Z", "+00:00", "-23:59", "+05:30"):
                lines.append('{"shipDate":"%04d-%02d-%02dT%02d:%02d:%02d%s%s","quantity":%d,"complete":%s}' % (y, rng.randrange(1, 13), rng.randrange(1, 29), rng.randrange(24), rng.randrange(60),
                             rng.randrange(60), frac, off, rng.choice([0, -1, 2147483647, -2147483648, 77]), rng.choice(["true", "false"])))
    cols = oracle.parse(ORDER, as_u8("\n".join(lines).encode()))
    assert cols.n_errors == 0
    write(writer, ORDER, cols, oracle.write(ORDER, cols, NDJSON, abi.PJ_INCLUDE_NON_NULL))
    rows = cols.arrays[COL["ord_ship_epoch"]].view(np.int64)
    nanos = cols.arrays[COL["ord_ship_nanos"]].view(np.int32)
    rows[3] = -10 ** 13; rows[5] = 10 ** 14; rows[9] = 2 ** 40; nanos[7] = -5  # what no parse gives
    write(writer, ORDER, cols, oracle.write(ORDER, cols, NDJSON, abi.PJ_INCLUDE_NON_NULL), recs=32)


def test_rows_in_another_order(writer, oracle):
    """A record map of the caller's own: rows shuffled, repeated or left out take the general road."""
    rng = np.random.default_rng(5)
    cols = oracle.parse(MIXED, pj.gen_text(MIXED, 7, 0, 200, ESC))
    kind = cols.arrays[COL["rec_type"]][:200]
    row = cols.arrays[COL["rec_row"]].view(np.uint32)[:200]
    for case in range(4):
        keep = kind.copy(), row.copy()
        if case == 0:
            p = rng.permutation(200); kind[:], row[:] = kind[p], row[p]
        elif case == 1:
            row[kind == 1] = row[kind == 1][0]
        elif case == 2:
            kind[50:90] = abi.PJ_TYPE_NONE
        else:
            kind[100:], row[100:] = keep[0][:100], keep[1][:100]
        write(writer, MIXED, cols, oracle.write(MIXED, cols, NDJSON, abi.PJ_INCLUDE_NON_NULL), recs=96)
        kind[:], row[:] = keep


def test_literals_out_of_range_and_present_bits(writer, oracle):
    """Enum values beyond the literals, booleans other than 0 and 1, list elements of a property that is not present."""
    cols = oracle.parse(PET, pj.gen_text(PET, 8, 0, 100, 0))
    cols.arrays[COL["pet_status"]][:100] = np.arange(100)
    cols.arrays[COL["pet_present"]][:100] = np.arange(100) % 64
    for inclusion in INCLUSIONS:
        write(writer, PET, cols, oracle.write(PET, cols, NDJSON, inclusion), inclusion=inclusion, recs=64)
    cols = oracle.parse(ORDER, pj.gen_text(ORDER, 8, 0, 100, 0))
    cols.arrays[COL["ord_complete"]][:100] = np.arange(100)
    write(writer, ORDER, cols, oracle.write(ORDER, cols, NDJSON, abi.PJ_INCLUDE_NON_NULL))


SIZES = [0, 1, 17, 255, 511, 512, 513, 1000, 2047, 2048, 2049, 4095, 4097, 33000]


def long_text(rng, n, dirty):
    """Pets whose strings and lists are as long as what warps take over, and a byte more or less."""
    word = lambda k: "".join(rng.choice(['\\"', "\\n", "\\u0001", "x"]) if rng.random() < dirty else "abcdefg"[j % 7] for j in range(k))
    out = []
    for i in range(n):
        urls = ",".join('"%s"' % word(rng.choice([0, 3, 30, 300, 1100])) for _ in range(rng.choice([0, 1, 7, 8, 9, 32, 33, 70])))
        tags = ",".join(rng.choice(["{}", '{"id":%d}' % j, '{"id":%d,"name":"%s"}' % (j, word(rng.choice([0, 9, 512, 2100])))]) for j in range(rng.choice([0, 1, 7, 8, 9, 40])))
        out.append('{"id":%d,"category":{"id":1,"name":"%s"},"name":"%s","photoUrls":[%s],"tags":[%s]}' % (i, word(rng.choice(SIZES[:-1])), word(rng.choice(SIZES)), urls, tags))
    return as_u8("\n".join(out).encode())


@pytest.mark.parametrize("dirty", [0, 0.002, 0.5])
@pytest.mark.parametrize("seed", range(3))
def test_long_strings_and_lists(writer, oracle, seed, dirty):
    """In the window, beyond it (one record after the other) and on the general road (no room to stage a tile, a record map of the caller's own)."""
    rng = random.Random(seed)
    cols = oracle.parse(PET, long_text(rng, 24, dirty))
    assert cols.n_errors == 0
    want = oracle.write(PET, cols, NDJSON, abi.PJ_INCLUDE_NON_NULL)
    for shape in [dict(recs=24, shared=131072), dict(recs=3, shared=100 * 1024, mis=3, order=5), dict(recs=1, shared=65536, mis=15), dict(recs=1, shared=131072, mis=1), dict(recs=24, shared=16384, mis=7), dict(recs=2, shared=8192)]:
        write(writer, PET, cols, want, **shape)
    mixed = oracle.parse(MIXED, np.concatenate([long_text(rng, 40, dirty), as_u8(b"\n"), pj.gen_text(MIXED, seed, 0, 40, ESC if dirty else 0)]))
    n = mixed.n_records
    kind, row = mixed.arrays[COL["rec_type"]][:n], mixed.arrays[COL["rec_row"]].view(np.uint32)[:n]
    kind[:], row[:] = kind[::-1].copy(), row[::-1].copy()
    want = oracle.write(MIXED, mixed, NDJSON, abi.PJ_INCLUDE_NON_NULL)
    for shape in [dict(recs=80, shared=100 * 1024, mis=5), dict(recs=16, shared=8192, order=3)]:
        write(writer, MIXED, mixed, want, **shape)


@pytest.mark.parametrize("length, esc", [(511, 0), (512, 0), (512, 40), (1000, 0), (5000, 30)])
def test_more_long_strings_than_a_tile_keeps(writer, oracle, length, esc):
    text = "".join('\\"' if esc and k % esc == 3 else "q" for k in range(length))
    line = lambda i: ('{"id":%d,' % i + ",".join('"%s":"%s%s"' % (k, text, "z" * (i % 5)) for k in ("username", "firstName", "lastName", "email", "password", "phone")) + "}").encode()
    cols = oracle.parse(USER, as_u8(b"\n".join(line(i) for i in range(70))))
    want = oracle.write(USER, cols, NDJSON, abi.PJ_INCLUDE_NON_NULL)
    for shape in [dict(recs=70, shared=131072), dict(recs=70, shared=16384, mis=9), dict(recs=40, shared=131072, mis=2, order=7), dict(recs=2, shared=80 * 1024), dict(recs=2, shared=65536)]:
        write(writer, USER, cols, want, **shape)


def test_a_window_holds_a_record(writer):
    """Of the average size, and one and a half; else the tile is made for the general road."""
    out = (C.c_uint32 * 2)()
    for per in [60, 300, 1800, 5000, 9000, 16000, 30000, 38000, 43000, 60000, 10 ** 6]:
        for model in (0, 2):
            for items in (0, 10, 200):
                rows = [0, 0, 0]
                rows[model] = n = 50_000
                writer.emu_write_shape(C.c_uint64(n), (C.c_uint64 * 3)(*rows), C.c_uint64(n * per), C.c_uint64(n * items if model == 0 else 0), C.c_uint64(0), out)
                staged, text = per + 40 + 8 * (items if model == 0 else 0), per + 130 + 3 * (items if model == 0 else 0)
                fits = staged * 1.04 + 1024 + 1.5 * text + 300 <= (128 if model == 0 and items > 16 else 100 if model == 0 else 64) * 1024
                assert out[1] >= out[0] * staged + 1.4 * text if fits else out[0] >= 16, (per, model, items, out[0], out[1])


def fall(off, row, by):
    """The range of string `row` goes back by `by` bytes: the string behind it shares them."""
    off[row + 1] = off[row] - by


@pytest.mark.parametrize("recs", [3, 32, 128])
def test_offsets_that_fall_where_no_string_is(writer, oracle, recs):
    """A string that is absent, or not written, may have any offsets: what two rows then share is escaped in both."""
    rng = random.Random(recs)
    esc = [b'\\"', b"\\n", b"\\u0001", b"x"]
    word = lambda k: b"".join(rng.choice(esc) for _ in range(k))
    # a table of Users: every string column falls at rows of its own
    n = 96
    keys = [b"username", b"firstName", b"lastName", b"email", b"password", b"phone"]
    cols = oracle.parse(USER, as_u8(b"\n".join(b'{"id":%d,%s}' % (i, b",".join(b'"%s":"%s"' % (k, word(12)) for k in keys)) for i in range(n))))
    present = cols.arrays[COL["usr_present"]]
    for f, name in enumerate(["username", "firstname", "lastname", "email", "password", "phone"]):
        off = cols.arrays[COL[f"usr_{name}_off"]].view(np.uint32)
        for row in range(1 + f, n - 1, 7):
            present[row] &= ~(2 << f) & 0xFF
            fall(off, row, 9)
    for inclusion in INCLUSIONS:
        write(writer, USER, cols, oracle.write(USER, cols, NDJSON, inclusion), inclusion=inclusion, recs=recs)
    # Pets: a category that is not there, a category's name, an element's name
    n = 64
    pet = b'{"id":%d,"category":{"id":1,"name":"%s"},"name":"%s","photoUrls":["%s"],"tags":[{"id":2,"name":"%s"},{"id":3,"name":"%s"}]}'
    for where in ("category", "category name", "name", "tag name", "photo"):
        cols = oracle.parse(PET, as_u8(b"\n".join(pet % ((i,) + tuple(word(12) for _ in range(5))) for i in range(n))))
        assert cols.n_errors == 0
        a = {k: cols.arrays[v] for k, v in COL.items() if k.startswith("pet_")}
        for row in range(1, n - 1, 5):
            if where == "category":
                a["pet_present"][row] &= ~2 & 0xFF
                fall(a["pet_cat_name_off"].view(np.uint32), row, 7)
            elif where == "category name":
                a["pet_cat_present"][row] &= ~2 & 0xFF
                fall(a["pet_cat_name_off"].view(np.uint32), row, 7)
            elif where == "name":
                a["pet_present"][row] &= ~4 & 0xFF
                fall(a["pet_name_off"].view(np.uint32), row, 7)
            elif where == "tag name":
                a["pet_tag_present"][2 * row] &= ~2 & 0xFF
                fall(a["pet_tag_name_off"].view(np.uint32), 2 * row, 7)
            else:
                a["pet_present"][row] &= ~8 & 0xFF
                fall(a["pet_photo_str_off"].view(np.uint32), row, 7)
        for inclusion in INCLUSIONS:
            write(writer, PET, cols, oracle.write(PET, cols, NDJSON, inclusion), inclusion=inclusion, recs=recs)


@pytest.mark.parametrize("recs", [40, 128])
@pytest.mark.parametrize("falls", [False, True])
def test_tiles_with_many_bytes_to_escape(writer, oracle, falls, recs):
    """More 16-byte blocks with one than a tile keeps: its strings are looked over one per lane. Whole words and ends of strings, plain and not."""
    rng = random.Random(recs)
    word = lambda k: "".join(rng.choice(['\\"', "\\n", "\\u0001", "\\\\"]) if rng.random() < 0.2 else "abcdefg"[j % 7] for j in range(k))
    length = lambda: rng.choice([0, 1, 2, 3, 4, 5, 7, 8, 9, 15, 16, 17, 31, 33, 63] + [511, 512, 513] * (recs < 100))
    users = ['{"id":%d,%s}' % (i, ",".join('"%s":"%s"' % (k, word(length())) for k in ("username", "firstName", "lastName", "email", "password", "phone"))) for i in range(150)]
    pets = ['{"id":%d,"category":{"id":1,"name":"%s"},"name":"%s","photoUrls":["%s","%s"],"tags":[{"id":2,"name":"%s"},{"name":"%s"}]}' % ((i,) + tuple(word(length()) for _ in range(6))) for i in range(150)]
    mixed = [x for pair in zip(users, pets) for x in pair]
    for schema, lines in ((USER, users), (PET, pets), (MIXED, mixed)):
        cols = oracle.parse(schema, as_u8("\n".join(lines)))
        assert cols.n_errors == 0
        if falls and schema != PET:
            for row in range(1, 149, 9):
                cols.arrays[COL["usr_present"]][row] &= ~2 & 0xFF
                off = cols.arrays[COL["usr_username_off"]].view(np.uint32)
                off[row + 1] = max(int(off[row]) - 5, 0)
        for inclusion in INCLUSIONS:
            want = oracle.write(schema, cols, NDJSON, inclusion)
            for shape in (dict(shared=131072), dict(shared=100 * 1024, mis=7, order=3)):
                write(writer, schema, cols, want, inclusion=inclusion, recs=recs, **shape)


@pytest.mark.parametrize("flags", [0, ESC | SPARSE, ZIPF | ESC])
def test_blocks_of_short_pets(writer, oracle, flags):
    """Half as many threads to a tile: whole tiles, lists, windows in rounds, the general road."""
    rng = random.Random(7)
    cols = oracle.parse(PET, pj.gen_text(PET, 12, 0, 300, flags))
    edges, long_ = oracle.parse(PET, edge_text(rng, 300)), oracle.parse(PET, long_text(rng, 12, 0.1))
    short = oracle.parse(PET, as_u8("\n".join('{"id":%d,"name":"%s","photoUrls":[]}' % (i, "ab"[: i % 3]) for i in range(600))))
    writer.emu_write_short(1)
    try:
        for c in (cols, edges, long_, short):
            want = oracle.write(PET, c, NDJSON, abi.PJ_INCLUDE_NON_NULL)
            for shape in (dict(recs=256, shared=131072), dict(recs=96, shared=28 * 1024, mis=9, order=3), dict(recs=5, shared=8192, mis=1)):
                write(writer, PET, c, want, **shape)
    finally:
        writer.emu_write_short(0)


def test_no_records(writer, oracle):
    cols = abi.HostColumns(PET, abi.default_caps(PET, 1, 16))
    n = C.c_uint64()
    assert writer.emu_write_tiles(PET, 0, 0, 0, C.byref(cols.raw), None, C.c_uint64(0), 32, 8192, 0, C.byref(n)) == 0 and n.value == 0


def test_columns_are_counted(writer):
    """The limits of the staging (a column per lane) are checked when the kernel is compiled, on a count of what it is given."""
    out = (C.c_uint32 * 4)()
    writer.emu_write_columns(out)
    assert tuple(out[:2]) == tuple(out[2:]) and 0 < out[0] <= 32 and 0 < out[1] <= 32 and out[0] + out[1] == len(abi.schema_columns(MIXED)) - 5


def test_shapes_fit(writer):
    out = (C.c_uint32 * 2)()
    for n in (0, 1, 20, 5000, 10 ** 6, 10 ** 8):
        for rows in ((n, 0, 0), (0, n, 0), (0, 0, n), (n // 3, n // 3, n // 3)):
            for per in (0, 30, 200, 3000, 10 ** 6):
                for items in (0, 3, 50, 10 ** 4):
                    writer.emu_write_shape(C.c_uint64(n), (C.c_uint64 * 3)(*rows), C.c_uint64(n * per), C.c_uint64(n * items), C.c_uint64(n * items), out)
                    assert 1 <= out[0] <= 256 and 8192 <= out[1] <= 128 * 1024


@pytest.mark.skipif(os.environ.get("PJ_EMU_SANITIZE") == "1", reason="is the run under the sanitizers")
def test_under_sanitizers():
    asan = subprocess.run(["gcc", "-print-file-name=libasan.so"], capture_output=True, text=True).stdout.strip()
    env = dict(os.environ, PJ_EMU_SANITIZE="1", LD_PRELOAD=asan, ASAN_OPTIONS="detect_leaks=0:detect_stack_use_after_return=0")
    r = subprocess.run([sys.executable, "-m", "pytest", "-q", "-x", "-p", "no:cacheprovider", __file__, "-k", "edges and 2 or dates or another_order or generated and 4"], env=env, capture_output=True, text=True, cwd=ROOT)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-3000:]
