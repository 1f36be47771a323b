"""k_parse_items (csrc/pj_item.cuh) run on the CPU, block by block, against the checker: no GPU needed.

tests/host_emu/pj_block_emu.h gives the kernel's source the threads, warp collectives and barriers of one block and reports lanes
that part at a collective, threads that part at a barrier and waits that do not end; one test repeats a slice of the others under
AddressSanitizer and UndefinedBehaviorSanitizer.
"""
import ctypes as C
import os
import random
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from pj_testlib import abi, as_u8, nrec_bound, pj, same_result
from test_host_emulation import blank_mutations
from test_oracle_crosscheck import mutate

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
NDJSON, ARRAY = abi.PJ_FRAMING_NDJSON, abi.PJ_FRAMING_ARRAY
PET, ORDER, USER, MIXED = abi.PJ_SCHEMA_PET, abi.PJ_SCHEMA_ORDER, abi.PJ_SCHEMA_USER, abi.PJ_SCHEMA_MIXED
ALL = abi.PJ_GEN_ESCAPES | abi.PJ_GEN_WHITESPACE | abi.PJ_GEN_MALFORMED | abi.PJ_GEN_SPARSE
FLAG_SETS = [0, abi.PJ_GEN_ESCAPES, abi.PJ_GEN_WHITESPACE, abi.PJ_GEN_MALFORMED, abi.PJ_GEN_SPARSE, ALL, abi.PJ_GEN_ZIPF_LISTS | ALL]


class Opts(C.Structure):
    _fields_ = [("len", C.c_uint64), ("slack", C.c_uint64), ("goff", C.c_uint64)] + [
        (k, C.c_uint32) for k in ("array", "is_first", "is_last", "opts", "tile_bytes", "win_bytes", "str_words", "row_cap", "order")] + [("rec_cap", C.c_uint64)]


@pytest.fixture(scope="session")
def emu():
    """The kernel for the host, a library per model set: {schema: CDLL}."""
    src = os.path.join(HERE, "host_emu", "pj_item_emu.cpp")
    csrc = os.path.join(ROOT, "micronaut3-bug_b200", "csrc")
    deps = [src, os.path.join(HERE, "host_emu", "pj_block_emu.h")] + [os.path.join(csrc, f) for f in os.listdir(csrc) if f.endswith((".cuh", ".h", ".inc"))]
    san = os.environ.get("PJ_EMU_SANITIZE") == "1"
    flags = ["-O1", "-g", "-fsanitize=address,undefined", "-fno-sanitize-recover=all"] if san else ["-O2"]

    def build(schema):
        lib = os.path.join(HERE, "host_emu", f"libpj_item_emu{schema}{'_san' if san else ''}.so")
        if not os.path.exists(lib) or any(os.path.getmtime(d) > os.path.getmtime(lib) for d in deps):
            subprocess.run(["g++", *flags, "-std=c++17", "-fno-extern-tls-init", "-fPIC", "-shared", "-w", f"-DEMU_SCHEMA={schema}", "-I", os.path.join(ROOT, "include"), "-I", csrc,
                            "-x", "c++", src, "-o", lib], check=True)
        cdll = C.CDLL(lib)
        cdll.emu_item_error.restype = C.c_char_p
        cdll.emu_item_barriers.restype = C.c_uint64
        return cdll

    with ThreadPoolExecutor() as pool:
        return dict(zip((1, 2, 3, 4), pool.map(build, (1, 2, 3, 4))))


class Run:
    """A parse by the emulated kernel: its columns, and what it says about itself."""

    def __init__(self, emu, schema, text, framing=NDJSON, tile=32768, slack=4096, mis=0, opts=0, order=0, str_words=None, row_cap=256, shard_slack=0,
                 is_first=1, is_last=1, goff=0):
        buf = as_u8(text)
        raw = np.full(buf.size + 64, 0xEE, np.uint8)
        at = (-raw.ctypes.data) % 16 + mis
        raw[at:at + buf.size] = buf
        self.cols = abi.HostColumns(schema, abi.default_caps(schema, nrec_bound(buf), buf.size), alloc=lambda nb: np.full(nb, 0xA5, np.uint8))
        win = min(tile + slack, 65536 - 64)
        o = Opts(len=buf.size - shard_slack, slack=shard_slack, goff=goff, array=framing == ARRAY, is_first=is_first, is_last=is_last, opts=opts, tile_bytes=tile,
                 win_bytes=win, str_words=str_words or win // 4, row_cap=row_cap, order=order, rec_cap=nrec_bound(buf))
        stats = (C.c_uint64 * 5)()
        lib = emu[schema]
        self.status = lib.emu_item_parse(C.byref(o), C.c_void_p(raw.ctypes.data + at), C.byref(self.cols.raw), stats)
        assert self.status >= 0, lib.emu_item_error().decode()
        self.fast, self.dense, self.longest, self.tiles, self.strs_per_kb = stats
        self.barriers = lib.emu_item_barriers()


SHAPES = [dict(), dict(tile=1024, slack=4096, mis=5), dict(tile=4096, slack=1024, mis=15, order=3), dict(tile=16384, slack=28672, str_words=3000, order=6)]


@pytest.mark.parametrize("schema", [PET, ORDER, USER, MIXED])
@pytest.mark.parametrize("flags", FLAG_SETS)
def test_generated_text(emu, oracle, schema, flags):
    text = pj.gen_text(schema, 0xE11, 0, 300, flags)
    want = oracle.parse(schema, text)
    for shape in SHAPES:
        got = Run(emu, schema, text, **shape)
        assert same_result(want, got.cols) == "", shape


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_mutated_text(emu, oracle, seed):
    rng = random.Random(seed)
    for it in range(60):
        schema = rng.choice([1, 1, 2, 3, 4, 4])
        lines = bytes(pj.gen_text(schema, rng.randrange(1 << 30), rng.randrange(1000), 40, rng.choice(FLAG_SETS))).split(b"\n")[:-1]
        out = [ln if rng.random() < 0.2 else mutate(rng, ln) for ln in lines]
        body = as_u8(blank_mutations(rng, b"\n".join(out)))
        opts = rng.choice([0, 0, 1, 2, 4, 7])
        got = Run(emu, schema, body, opts=opts, **rng.choice(SHAPES))
        assert same_result(oracle.parse(schema, body, opts=opts), got.cols) == "", (seed, it, schema, opts)


def test_mutated_arrays(emu, oracle):
    rng = random.Random(9)
    for it in range(60):
        schema = rng.choice([1, 2, 3, 4])
        text = bytes(pj.gen_text(schema, rng.randrange(1 << 30), 0, 40, abi.PJ_GEN_ARRAY | rng.choice(FLAG_SETS[:6])))
        if it % 3:
            text = mutate(rng, text)
        want = oracle.parse(schema, as_u8(text), ARRAY)
        got = Run(emu, schema, text, ARRAY, **rng.choice(SHAPES))
        assert same_result(want, got.cols) == "", (it, schema)
        assert (want.raw.doc_err_kind, want.raw.doc_err_off) == (got.cols.raw.doc_err_kind, got.cols.raw.doc_err_off)


def test_shards(emu, oracle):
    """Cut anywhere, with the bytes behind as slack: every record is parsed by the shard that owns the line feed before it."""
    rng = random.Random(11)
    text = as_u8(blank_mutations(rng, pj.gen_text(PET, 3, 0, 300, ALL).tobytes()))
    want = oracle.parse(PET, text)
    for parts in (2, 5):
        cuts = [text.size * k // parts for k in range(parts + 1)]
        n = 0
        for k in range(parts):
            lo, hi = cuts[k], cuts[k + 1]
            slack = min(65536, text.size - hi)
            piece = text[lo:hi + slack]
            kw = dict(is_first=int(k == 0), is_last=int(hi + slack == text.size), goff=lo)
            got = Run(emu, PET, piece, tile=4096, mis=k, shard_slack=slack, **kw)
            assert same_result(oracle.parse(PET, piece, slack=slack, **kw), got.cols) == "", (parts, k)
            n += got.cols.n_records
        assert n == want.n_records


def test_known_answers(emu, oracle):
    from golden.kat_cases import CASES, OPTION_CASES
    from pj_testlib import SCHEMA_BY_NAME, records

    for name, schema, framing, data, expected in CASES:
        sch, fr = SCHEMA_BY_NAME[schema], ARRAY if framing == "array" else NDJSON
        got = Run(emu, sch, data, fr, tile=1024)
        assert same_result(oracle.parse(sch, as_u8(data), fr), got.cols) == "", name
    for name, schema, opts, data, expected in OPTION_CASES:
        sch = SCHEMA_BY_NAME[schema]
        assert records(Run(emu, sch, data, opts=opts).cols.as_dict(), sch) == expected, name


def test_keys_spelled_with_escapes(emu, oracle):
    """The text of a key decoded in place is followed by the bytes it freed, not by its closing quote."""
    u = lambda name, k: name[:k] + "\\u%04x" % ord(name[k]) + name[k + 1:]
    pet = ["id", "name", "photoUrls", "status", "category", "tags"]
    lines = ['{"%s":%d,"name":"a","photoUrls":["x"]}' % (u("id", k), 7 + k) for k in (0, 1)]
    for name in pet:  # every property, its first and last letter
        for k in (0, len(name) - 1):
            rec = '{"id":5,"name":"n","photoUrls":["p"],"category":{"id":1,"name":"c"},"tags":[{"id":2,"name":"t"}],"status":"sold"}'
            lines.append(rec.replace('"%s":' % name, '"%s":' % u(name, k)))
    lines += ['{"\\u0069ds":4,"name":"a","photoUrls":[]}', '{"\\u0069":4,"name":"a","photoUrls":[]}', '{"i\\/":4,"name":"a","photoUrls":[]}']  # names of nothing
    for line in lines:  # each on its own: a record for the exact parser takes its tile along
        body = as_u8(line + "\n")
        for schema in (PET, MIXED):
            want = oracle.parse(schema, body)
            assert want.n_errors == 0 and same_result(want, Run(emu, schema, body).cols) == "", line


@pytest.mark.parametrize("schema", [PET, ORDER, USER, MIXED])
def test_tile_shape_fits_shared_memory(emu, schema):
    """Every shape a call can get fits the kernel's shared memory and 16-bit window offsets; calls of few tiles get one resident block
    for each of them. (One record of 23 KB in an earlier call made a later one of 16 MB ask for 211 KB of 200.)"""
    out = (C.c_uint32 * 7)()
    guess = [0, 300, 146, 190, 230][schema]
    lens = [0, 1, 300, 5000, 10**5] + [int(10**5 * 1.21 ** k) for k in range(1, 60)] + list(range(15_000_000, 17_000_000, 40_000))
    for avg in [0, 1, 9, 40, 146, 200, 230, 250, 300, 700, 2000, 9000, 20_000, 10**6]:
        for longest in [0, 300, 3277, 9000, 22_000, 22_886, 23_000, 65_000, 1 << 30]:
            for tile_opt, strs in ((0, 0), (0, 100), (0, 250), (0, 400), (1, 0), (4096, 0), (20_000, 0), (20_000, 300), (32_768, 0), (1 << 20, 400)):
                for n in lens if tile_opt == 0 and strs == 0 else lens[:40:8]:
                    emu[schema].emu_item_shape(C.c_uint64(n), C.c_double(avg), C.c_double(guess), C.c_uint32(longest), C.c_uint32(strs), C.c_uint32(tile_opt), out)
                    tile, win, words, rows, total, most, blocks = out
                    where = (n, avg, longest, strs, tile_opt, list(out))
                    assert total <= most, where
                    assert 1024 <= tile <= 36864 and tile % 32 == 0 and tile < win <= 65536 - 64 and win % 16 == 0, where
                    assert 24 <= rows <= 256 and words * 9 + 9 > win, where
                    if strs and tile_opt == 0 and longest <= 3277 and avg <= 300:  # a tile's strings have their words and are no more than its limit
                        assert words >= win * strs // 1024 + 2 and tile * strs // 1024 < 4096, where
                    if tile_opt == 0 and strs <= 100 and longest <= 3277 and avg <= 300:
                        assert blocks == 3, where


@pytest.mark.parametrize("part", [1, 2, 6])
def test_tiles_full_of_strings_beyond_ascii(emu, oracle, part):
    """Names in another script, slashes written as \\/: however many strings of a tile take a closer look, no record is left to the exact parser."""
    words = ["\u0438\u043c\u044f", "\u540d\u524d", "a\\/b\\/c", "\\u00e9t\\u00e9", "na\u00efve", "\\n"]
    keys = ["username", "firstName", "lastName", "email", "password", "phone"]
    lines = ['{"id":%d,%s,"userStatus":1}' % (i, ",".join('"%s":"%s%d"' % (k, words[(i + j) % 6] if j < part else "x", i) for j, k in enumerate(keys))) for i in range(400)]
    body = as_u8("\n".join(lines) + "\n")
    want = oracle.parse(USER, body)
    for tile in (32768, 16384):
        got = Run(emu, USER, body, tile=tile)
        assert same_result(want, got.cols) == "" and got.fast == want.n_records == 400


UNUSUAL = [b'"price":1.5,', b'"x":{"a":[1,{"b":"c"}],"d":"e"},', b'"x":["y",{"z":[]}],', b'"id":3,', b'"x":1e3,']  # valid, and only the exact parser knows them


@pytest.mark.parametrize("schema", [PET, ORDER, USER, MIXED])
@pytest.mark.parametrize("every", [1, 2, 7, 31, 90])
def test_unusual_records_stand_apart(emu, oracle, schema, every):
    """A valid record that only the exact parser knows is written by it alone, between the columns of its neighbours, whatever else its lines hold."""
    for flags in (0, ALL, abi.PJ_GEN_ZIPF_LISTS | abi.PJ_GEN_ESCAPES):
        lines = bytes(pj.gen_text(schema, every + flags, 0, 300 if not flags & abi.PJ_GEN_ZIPF_LISTS else 60, flags)).split(b"\n")[:-1]
        out = [ln[:1 + ln.index(b"{")] + UNUSUAL[(i // every) % len(UNUSUAL)] + ln[1 + ln.index(b"{"):] if i % every == every - 1 and b'":' in ln else ln for i, ln in enumerate(lines)]
        for framing, body in ((NDJSON, b"\n".join(out) + b"\n"), (ARRAY, b"[" + b",".join(out) + b"]")):
            body = as_u8(body)
            want = oracle.parse(schema, body, framing)
            for kw in (dict(), dict(tile=4096, mis=3, order=5)):
                got = Run(emu, schema, body, framing, **kw)
                assert same_result(want, got.cols) == "", (flags, framing, kw)
                if flags == 0 and framing == NDJSON:
                    assert got.fast >= want.n_records - want.n_errors - len(out) // every


def test_strings_too_long_for_a_reference_stand_apart(emu, oracle):
    long = '{"id":1,"username":"%s","phone":"5"}' % ("y" * 33000)
    users = ['{"id":%d,"username":"u%d"}' % (i, i) for i in range(60)]
    body = as_u8("\n".join(users[:30] + [long] + users[30:]) + "\n")
    got = Run(emu, USER, body, tile=16384, slack=45000)
    assert same_result(oracle.parse(USER, body), got.cols) == "" and got.fast >= 59
    pet = '{"id":1,"name":"n","photoUrls":["a"],"tags":[{"name":"%s"},{"id":2,"name":"t"}]}'
    body = as_u8("\n".join(pet % ("t" * (5000 if i == 20 else 5)) for i in range(40)) + "\n")
    got = Run(emu, PET, body, tile=16384, slack=8000)
    assert same_result(oracle.parse(PET, body), got.cols) == "" and got.fast >= 36  # (four lines are looked at together)


def test_documents_that_are_not_one_array(emu, oracle):
    """A text cut off in transfer, something behind the array, several arrays, extents without a value: the records are decoded as those of a
    clean document."""
    rng = random.Random(31)
    for schema in (PET, USER, MIXED):
        text = bytes(pj.gen_text(schema, 77, 0, 150, abi.PJ_GEN_ARRAY | abi.PJ_GEN_SPARSE))
        recs = text[1:-1]
        docs = [text[:cut] for cut in [1, 2, len(text) - 1] + [rng.randrange(len(text)) for _ in range(40)]]
        docs += [text + t for t in (b"]", b"x", b" \n", b",", b"[]", b'"', b"[" + recs + b"]", b',"a"', b" null ", b"}")]
        docs += [t + text for t in (b" ", b"x", b"[],", b"{}", b"]", b'"a"')]
        docs += [b"[" + recs + t + b"]" for t in (b",", b",,", b", ,{}", b"}", b"]", b"},{")] + [b"[ ]", b"[", b"[,]", b"[,,]", b"", b" ", b"[{}] [{}]", b"[{}][ ]", b"{},{}"]
        docs += [text.replace(b"},{\"id", b"}, \t,{\"id", 5), text.replace(b"},{\"id", b"}]],{\"id", 1), text.replace(b"},{\"id", b'}],"[",[{"id', 2)]
        for doc in docs:
            body = as_u8(doc)
            want = oracle.parse(schema, body, ARRAY)
            for kw in (dict(), dict(tile=2048, mis=9, order=2)):
                got = Run(emu, schema, body, ARRAY, **kw)
                assert same_result(want, got.cols) == "", (schema, doc[-60:], kw)
                assert (want.raw.doc_err_kind, want.raw.doc_err_off) == (got.cols.raw.doc_err_kind, got.cols.raw.doc_err_off), (schema, doc[-60:])
                assert got.fast >= (want.n_records - want.n_errors) - 2, (schema, doc[-60:], got.fast, want.n_records)


def test_the_first_value_of_a_repeated_key_is_judged(emu, oracle):
    """A failure there comes before everything else of the record, also when the repetition itself is not the first failure."""
    for first in ("1x2", "1.5", "null", "3", '"a"', "true", "[1]", "1" * 30, ""):
        for between in ('"category":"c"', '"category":7', '"name":5', '"name":"n"', '"name":"n" "x"'):
            for second in ("4", "null", "x", '"b"'):
                for status in ("", ',"status":"gone","status":"sold"', ',"status":null,"status":"gone"'):
                    line = '{"id":%s,%s,"id":%s%s,"name":"a","photoUrls":[]}' % (first, between, second, status)
                    body = as_u8(line + "\n")
                    want = oracle.parse(PET, body)
                    for order in (0, 1):
                        assert same_result(want, Run(emu, PET, body, tile=1024, order=order).cols) == "", line


@pytest.mark.parametrize("schema", [PET, USER, MIXED])
def test_records_longer_than_the_window(emu, oracle, schema):
    """They are the exact parser's, where they lie; the records beside them in their tile are not."""
    rng = random.Random(schema)
    pad = "".join('"%s",' % ("p%d" % i * 3 + ("\\n" if i % 9 == 0 else "") + ("\u00e9" if i % 11 == 0 else "")) for i in range(1500))
    pet = '{"id":1,"name":"n","photoUrls":[%s"z"],"tags":[{"id":2,"name":"t"}]%s}'
    user = '{"id":1,"username":"%s","phone":"5"%s}'
    longs = [pet % (pad, e) if schema != USER else user % ("u" * 9000 + "\\n" * 1500, e) for e in ("", ',"status":"gone"', ',"x":[1.5]', ' } ', '', ',"id":')]
    longs += [" " * 12000, " " * 9000 + "{}", '{"x":"' + "y" * 9000]
    for n, where in ((40, "middle"), (3, "first"), (3, "last"), (0, "alone")):
        for long in longs:
            lines = bytes(pj.gen_text(schema, 5, 0, n, 0)).decode().split("\n")[:-1]
            lines.insert({"middle": n // 2, "first": 0}.get(where, len(lines)), long)
            for framing, text in ((NDJSON, "\n".join(lines) + rng.choice(["", "\n"])), (ARRAY, "[" + ",".join(lines) + "]")):
                body = as_u8(text)
                want = oracle.parse(schema, body, framing)
                for kw in (dict(tile=4096, slack=1024, mis=3), dict(tile=1024, slack=4096, order=7), dict(tile=16384, slack=2048, mis=8, order=3)):
                    got = Run(emu, schema, body, framing, **kw)
                    assert same_result(want, got.cols) == "", (where, long[-40:], framing, kw)
                    assert (want.raw.doc_err_kind, want.raw.doc_err_off) == (got.cols.raw.doc_err_kind, got.cols.raw.doc_err_off)
                    assert got.fast >= want.n_records - want.n_errors - 1


def test_lines_that_end_inside_a_string(emu, oracle):
    """However many they are, the index takes a fixed number of rounds (it closed one of them in each)."""
    rng = random.Random(4)
    for line in ('"', '{"id', '{"id":1,"username":"a', '{"id":1,"username":"a","phone":"x\\"', '{"id":"7","username":"a"}"'):
        for share in (1.0, 0.5, 0.03):
            text = "\n".join(line if rng.random() < share else '{"id":2,"username":"b"}' for _ in range(3000))
            body = as_u8(text)
            want = oracle.parse(USER, body)
            for kw in (dict(tile=4096), dict(tile=32768, mis=7, order=9)):
                got = Run(emu, USER, body, **kw)
                assert same_result(want, got.cols) == "", (line, share, kw)
                assert got.barriers <= 120 * got.tiles, (line, share, kw, got.barriers, got.tiles)


@pytest.mark.parametrize("schema", [PET, ORDER, USER, MIXED])
def test_tiles_with_more_lines_or_strings_than_room(emu, oracle, schema):
    """Their lines are sized and written where they lie, by either parser, up to the last bytes of the input and of a shard's slack."""
    rng = random.Random(schema)
    flags = ALL | (abi.PJ_GEN_ZIPF_LISTS if schema in (PET, MIXED) else 0)
    for it in range(12):
        lines = bytes(pj.gen_text(schema, it, 0, 60, rng.choice([0, flags]))).split(b"\n")[:-1]
        lines = [mutate(rng, ln) if rng.random() < 0.2 else ln for ln in lines] + [b'{"id":1}', b'{"x":[1],"id":2}', b"{}", b" "][: it % 5]
        rng.shuffle(lines)
        for room in (dict(row_cap=3), dict(str_words=20)):
            opts = rng.choice([0, 1, 2, 4])
            for framing, text in ((NDJSON, b"\n".join(lines) + rng.choice([b"", b"\n", b"\n" + b" " * 40])), (ARRAY, b"[" + b",".join(lines) + b"]" + b" " * (it * 5))):
                body = as_u8(text)
                got = Run(emu, schema, body, framing, tile=4096, mis=it, opts=opts, **room)
                assert same_result(oracle.parse(schema, body, framing, opts=opts), got.cols) == "", (it, room, framing)
            body = as_u8(b"\n".join(lines) + b"\n")
            cut = body.size // 2
            got = Run(emu, schema, body, tile=4096, shard_slack=body.size - cut, is_last=0, **room)
            assert same_result(oracle.parse(schema, body, slack=body.size - cut, is_last=0), got.cols) == "", (it, room)


def test_lists_of_short_strings_fit_once_seen(emu, oracle):
    """More strings than a window's usual room: the kernel says how many there are, and the shape made of that holds them."""
    lines = ['{"id":%d,"name":"n","photoUrls":[%s]}' % (i, ",".join('"a%d"' % k for k in range(40))) for i in range(500)]
    body = as_u8("\n".join(lines) + "\n")
    want = oracle.parse(PET, body)
    out = (C.c_uint32 * 7)()
    strs, fast = 0, []
    for _ in range(3):
        emu[PET].emu_item_shape(C.c_uint64(10**9), C.c_double(body.size / 500), C.c_double(300), C.c_uint32(280), C.c_uint32(strs), C.c_uint32(0), out)
        got = Run(emu, PET, body, tile=out[0], slack=out[1] - out[0], str_words=out[2], row_cap=out[3])
        assert same_result(want, got.cols) == ""
        strs = got.strs_per_kb
        fast.append(got.fast)
    assert fast[0] < 250 and fast[1] == fast[2] == 500, (fast, strs)


# kinds of text: milliseconds per 19 MB with k_parse_stream / k_parse_items, share of fast and dense records each reports, longest record
KINDS = {"plain": ((0.050, 1.0, 1.0), (0.062, 1.0, 1.0), 250), "spaced": ((0.195, 1.0, 0.1), (0.089, 1.0, 0.0), 400), "script": ((0.084, 1.0, 0.1), (0.114, 1.0, 1.0), 250),
         "nested": ((0.340, 0.0, 0.0), (0.740, 0.0, 0.0), 300), "unknown": ((0.344, 0.0, 0.0), (0.130, 1.0, 0.0), 300), "long": ((0.5, 1.0, 0.0), (15.6, 0.0, 0.0), 40000)}
BEST = {"plain": 0, "spaced": 1, "script": 0, "nested": 0, "unknown": 1, "long": 0}


def choose(emu, calls, size=19_000_000):
    """The kernel each of the calls took: 0 a record per thread, 1 k_parse_items."""
    lib = emu[PET]
    lib.emu_choice_reset()
    took, now = [], 0
    for kind in calls:
        took.append(now)
        (ms, fast, dense), longest = KINDS[kind][now], KINDS[kind][2]
        n = size // longest
        now = lib.emu_choice_note(C.c_uint64(size), C.c_float(ms * size / 19e6), C.c_uint64(n), C.c_uint64(0), C.c_uint64(int(n * fast)), C.c_uint64(int(n * dense)), C.c_uint32(longest))
    return took


def test_choice_of_the_kernel(emu):
    """It settles on the faster kernel for every kind of text, also after other kinds, and text that goes back and forth does not drag it along."""
    for kind in KINDS:
        took = choose(emu, [kind] * 500)
        assert sum(t != BEST[kind] for t in took) <= 10, kind  # of 500
        assert choose(emu, [kind] * 8)[3:] == [BEST[kind]] * 5, kind
        for before in KINDS:
            took = choose(emu, [before] * 6 + [kind] * (12 if (before, kind) != ("nested", "unknown") else 80))  # (those two look the same to k_parse_stream)
            assert took[-4:] == [BEST[kind]] * 4, (before, kind, took)
    assert sum(choose(emu, ["long"] * 10)) == 0  # records that fill a window are not even tried
    took = choose(emu, ["spaced", "plain"] * 200)
    assert sum(a != b for a, b in zip(took, took[1:])) <= 16
    assert choose(emu, ["plain", "spaced", "spaced"] + ["plain"] * 100)[-1] == 0  # it does not stay for good
    assert choose(emu, ["spaced"] * 5, size=20_000) == [0, 1, 1, 1, 1]  # too short to be timed: by the spelling alone


@pytest.mark.parametrize("first, later, other, best", [(0.255, 0.113, 0.172, 0), (0.255, 0.113, 0.080, 1), (0.60, 0.46, 0.35, 1)])
def test_a_handles_first_call_does_not_decide_alone(emu, first, later, other, best):
    """k_parse_stream's first call on a handle takes longer: where it loses narrowly it has a second one, then the faster kernel stays."""
    lib, size, took, now, runs = emu[USER], 5_000_000, [], 0, 0
    lib.emu_choice_reset()
    for _ in range(40):
        took.append(now)
        ms = other if now else (later if runs else first)
        runs += not now
        now = lib.emu_choice_note(C.c_uint64(size), C.c_float(ms), C.c_uint64(50_000), C.c_uint64(0), C.c_uint64(0), C.c_uint64(0), C.c_uint32(110))
    assert took[:3] == [0, 1, 0 if first - other < 0.2 else 1] and took[3:] == [best] * 37, took


def test_under_sanitizers():
    asan = subprocess.run(["gcc", "-print-file-name=libasan.so"], capture_output=True, text=True).stdout.strip()
    if not os.path.isabs(asan) or not os.path.exists(asan):
        pytest.skip("no libasan beside this gcc")
    env = dict(os.environ, PJ_EMU_SANITIZE="1", LD_PRELOAD=asan, ASAN_OPTIONS="detect_leaks=0:abort_on_error=0:detect_stack_use_after_return=0", UBSAN_OPTIONS="print_stacktrace=1")
    r = subprocess.run([sys.executable, "-m", "pytest", "-x", "-q", "-p", "no:cacheprovider", os.path.abspath(__file__), "-k", "not sanitizers and not (mutated_text and 3)"],
                       env=env, capture_output=True, text=True, cwd=HERE, timeout=1500)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-3000:]
    assert "passed" in r.stdout
