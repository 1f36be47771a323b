"""The kernel that spreads a tile over strings (k_parse_items) at the sizes where it can go wrong, against the checker."""
import random

import pytest

from pj_testlib import abi, as_u8, pj, same_result
from test_gpu_parity import ARRAY, NDJSON, gpu_parse_device, gpu_parse_host

pytestmark = pytest.mark.gpu

SPACED = abi.PJ_GEN_WHITESPACE | abi.PJ_GEN_SPARSE


@pytest.fixture(scope="module")
def items_ctx():
    """A context whose NDJSON calls all take the kernel."""
    with pj.Context(device=0, flags=abi.PJ_OPT_TEST_ITEMS) as c:
        yield c


def parse(ctx, schema, body, framing=NDJSON, offset=0):
    """gpu_parse_device() by this kernel."""
    got = gpu_parse_device(ctx, schema, body, framing, offset)
    assert ctx.stats().stage_launches[3] == ctx.stats().stage_launches[2] > 0
    return got


def corpus(schema, n, kind):
    flags = {"plain": 0, "blanks": SPACED, "escapes": abi.PJ_GEN_ESCAPES, "broken": abi.PJ_GEN_MALFORMED | abi.PJ_GEN_WHITESPACE,
             "lists": abi.PJ_GEN_ZIPF_LISTS | abi.PJ_GEN_ESCAPES}[kind]
    lines = bytes(pj.gen_text(schema, 100 + n, 0, n, flags)).split(b"\n")[:-1]
    rng = random.Random(n)
    if kind == "blanks":  # lines that are no records, records without a string, unknown properties
        lines = [x for ln in lines for x in ((ln, b" \t") if rng.random() < 0.1 else (ln,))]
        lines += [b"{}", b'{"other":[1,{"a":"b"}],"id":7}', b'{"other":"x","id":8}']
    return b"\n".join(lines) + (b"\n" if n % 2 else b"")


@pytest.mark.parametrize("schema", [1, 2, 3, 4])
@pytest.mark.parametrize("kind", ["plain", "blanks", "escapes", "broken", "lists"])
@pytest.mark.parametrize("n", [1, 31, 33, 255, 257, 2000])
def test_groups_of_lines(items_ctx, oracle, schema, kind, n):
    body = as_u8(corpus(schema, n, kind))
    assert same_result(oracle.parse(schema, body, NDJSON), parse(items_ctx, schema, body, NDJSON, n % 16)) == ""


@pytest.mark.parametrize("n", [1, 32, 257, 3000])
def test_array_extents(items_ctx, oracle, n):
    body = pj.gen_text(1, 9 + n, 0, n, abi.PJ_GEN_ARRAY | abi.PJ_GEN_ESCAPES)
    assert same_result(oracle.parse(1, body, ARRAY), parse(items_ctx, 1, body, ARRAY)) == ""


def test_both_kernels_agree(items_ctx, oracle):
    body = pj.gen_text(4, 21, 0, 5000, 0)
    want = oracle.parse(4, body)
    with pj.Context(device=0, flags=abi.PJ_OPT_TEST_RECORDS) as records:
        assert same_result(want, gpu_parse_device(records, 4, body)) == "" and records.stats().stage_launches[3] == 0
    assert same_result(want, parse(items_ctx, 4, body)) == ""


def test_a_new_context_finds_its_kernel(oracle):
    """The first call takes the kernel with a record per thread; spaced text goes over to the other one, compact text comes back."""
    took = []
    with pj.Context(device=0) as c:
        for flags in (SPACED, SPACED, SPACED, 0, 0, 0):
            body = pj.gen_text(3, 4, 0, 1000, flags)
            assert same_result(oracle.parse(3, body), gpu_parse_device(c, 3, body)) == ""
            took.append(c.stats().stage_launches[3])
    assert took == [0, 1, 1, 1, 0, 0], took


@pytest.mark.parametrize("schema", [1, 2, 3, 4])
def test_unusual_records(items_ctx, oracle, schema):
    """Records that stand apart, keys in escapes, strings in another script, lines that end in a string, long records: by the kernel's own steps."""
    lines = bytes(pj.gen_text(schema, 8, 0, 3000, abi.PJ_GEN_SPARSE)).split(b"\n")[:-1]
    extra = [b'"x":{"a":[1,2.5]},', b'"\\u0069d":4,', '"y":"\u540d\u524d \\\\",'.encode(), b'"x":1.5,', b'"id":1,', b'"z":"a\\/b",']
    text = [ln[:1] + extra[i % 6] + ln[1:] if i % 5 == 0 else (ln[: len(ln) // 2] if i % 97 == 0 else ln) for i, ln in enumerate(lines)]
    text[1500:1500] = [b'{"id":1,"x":"' + b"y" * 90_000 + b'"}', b'{"id":1,"x":["' + b'","'.join([b"u" * 9] * 9000) + b'"]}']
    for framing, body in ((NDJSON, b"\n".join(text)), (ARRAY, b"[" + b",".join(t for t in text if t.endswith(b"}")) + b"]"), (ARRAY, b"[" + b",".join(lines)), (ARRAY, b"[" + b",".join(lines) + b",] x")):
        body = as_u8(body)
        want = oracle.parse(schema, body, framing)
        for _ in range(2):
            assert same_result(want, parse(items_ctx, schema, body, framing, 3)) == ""


def test_strings_beyond_ascii_and_short_ones_are_the_kernels_own(items_ctx, oracle):
    keys = ["username", "firstName", "lastName", "email", "password", "phone"]
    users = "\n".join('{"id":%d,%s}' % (i, ",".join('"%s":"\u0438\u043c\u044f\\n%d"' % (k, i) for k in keys)) for i in range(5000)).encode()
    pets = "\n".join('{"id":%d,"name":"n","photoUrls":[%s]}' % (i, ",".join('"a%d"' % k for k in range(40))) for i in range(5000)).encode()
    for schema, body in ((3, as_u8(users)), (1, as_u8(pets))):
        want = oracle.parse(schema, body)
        for _ in range(3):
            assert same_result(want, parse(items_ctx, schema, body)) == ""
        assert items_ctx.stats().fast_records == want.n_records == 5000  # (from the second call on, where there are more strings than usual)


def test_shards_pieces_and_ranges(oracle):
    """Cut lines, and launches that start from the totals of the one before."""
    text = as_u8(corpus(4, 4000, "blanks") + b"\n" + corpus(4, 3000, "broken"))
    want = oracle.parse(4, text)
    for kw in (dict(host_piece_bytes=50_000), dict(device_piece_bytes=150_001)):
        with pj.Context(device=0, flags=abi.PJ_OPT_TEST_ITEMS, **kw) as c:
            got = gpu_parse_host(c, 4, text) if "host_piece_bytes" in kw else gpu_parse_device(c, 4, text)
            assert same_result(want, got) == "" and c.stats().pieces > 3 and c.stats().stage_launches[3] == c.stats().pieces


def test_one_long_record_then_a_call_of_few_tiles(oracle):
    """The tile shape of a call of 16 MB whose context has seen a record of 25 KB: it asked for more shared memory than there is."""
    text = bytes(pj.gen_text(3, 5, 0, 83_000, abi.PJ_GEN_ARRAY))
    body = as_u8(text[:-1] + b',{"id":1,"username":"' + b"u" * 25_000 + b'"}]')
    assert 15_400_000 < body.size < 16_200_000
    want = oracle.parse(3, body, ARRAY)
    with pj.Context(device=0) as c:
        for _ in range(3):
            assert same_result(want, gpu_parse_device(c, 3, body, ARRAY)) == ""


def long_pets(n, name):
    return b"\n".join(b'{"id":%d,"name":"%s","photoUrls":["u%d"]}' % (i, b"n" * (name + i % 7), i) for i in range(n))


@pytest.mark.parametrize("offset", [0, 5])
@pytest.mark.parametrize("name", [16_400, 40_000])
def test_long_records_of_several_models_are_put_aside(oracle, name, offset):
    """A fresh context's first call on them does not wait for the kernel it starts with; the third in a row does not ask any more; usual records have it again."""
    long_ = as_u8(long_pets(40, name))
    usual = pj.gen_text(4, 11, 0, 20_000, abi.PJ_GEN_MALFORMED)
    took = []
    with pj.Context(device=0) as c:
        for body in (long_, long_, long_, usual, usual):
            assert same_result(oracle.parse(4, body), gpu_parse_device(c, 4, body, NDJSON, offset)) == ""
            s = c.stats()
            took.append((s.stage_launches[2], s.stage_launches[3]))
    assert took == [(2, 1), (2, 1), (1, 0), (1, 0), (1, 1)], took


@pytest.mark.parametrize("kw", [dict(host_piece_bytes=1 << 18), dict(device_piece_bytes=300_001)])
def test_long_records_in_pieces(oracle, kw):
    body = as_u8(long_pets(60, 30_000) + b"\n" + bytes(pj.gen_text(4, 5, 0, 4, 0)))
    with pj.Context(device=0, **kw) as c:
        for _ in range(2):
            got = gpu_parse_host(c, 4, body) if "host_piece_bytes" in kw else gpu_parse_device(c, 4, body, NDJSON, 3)
            assert same_result(oracle.parse(4, body), got) == ""
            s = c.stats()
            assert s.pieces > 1 and s.stage_launches[3] == (0 if "host_piece_bytes" in kw else s.pieces)


def test_few_bytes_of_several_models(items_ctx, oracle):
    """Around the input size that is looked at; one line, and line feeds only."""
    with pj.Context(device=0) as c:
        for body in (b"\n" * 16_383, b"\n" * 16_384, b" " * 16_384, long_pets(1, 16_384), long_pets(1, 16_300), long_pets(1, 300_000)):
            for off in (0, 1, 15):
                assert same_result(oracle.parse(4, as_u8(body)), gpu_parse_device(c, 4, body, NDJSON, off)) == ""
            assert same_result(oracle.parse(4, as_u8(body)), gpu_parse_host(c, 4, body)) == ""
