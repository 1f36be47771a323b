"""The kernel that spreads a tile over strings (k_parse_items) at the sizes where it can go wrong, against the checker."""
import random

import pytest

from pj_testlib import abi, as_u8, pj, same_result
from test_gpu_parity import ARRAY, NDJSON, gpu_parse_device

pytestmark = pytest.mark.gpu

SPACED = abi.PJ_GEN_WHITESPACE | abi.PJ_GEN_SPARSE


@pytest.fixture(scope="module")
def items_ctx():
    """A context whose NDJSON calls have gone over to the kernel for good: its texts changed their spelling twice."""
    c = pj.Context(device=0)
    for schema in (1, 2, 3, 4):
        for flags in (SPACED, 0, SPACED):
            gpu_parse_device(c, schema, pj.gen_text(schema, 3, 0, 400, flags))
    yield c
    c.close()


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
    assert same_result(oracle.parse(schema, body, NDJSON), gpu_parse_device(items_ctx, schema, body, NDJSON, n % 16)) == ""


@pytest.mark.parametrize("n", [1, 32, 257, 3000])
def test_array_extents(items_ctx, oracle, n):
    body = pj.gen_text(1, 9 + n, 0, n, abi.PJ_GEN_ARRAY | abi.PJ_GEN_ESCAPES)
    assert same_result(oracle.parse(1, body, ARRAY), gpu_parse_device(items_ctx, 1, body, ARRAY)) == ""


def test_both_kernels_agree(items_ctx, oracle):
    """The same text by a new context (a record per thread) and by one that has seen blanks."""
    body = pj.gen_text(4, 21, 0, 5000, 0)
    fresh = pj.Context(device=0)
    want = oracle.parse(4, body)
    assert same_result(want, gpu_parse_device(fresh, 4, body)) == "" and same_result(want, gpu_parse_device(items_ctx, 4, body)) == ""
    fresh.close()


def test_one_long_record_then_a_call_of_few_tiles(oracle):
    """The tile shape of a call of 16 MB whose context has seen a record of 25 KB: it asked for more shared memory than there is."""
    text = bytes(pj.gen_text(3, 5, 0, 83_000, abi.PJ_GEN_ARRAY))
    body = as_u8(text[:-1] + b',{"id":1,"username":"' + b"u" * 25_000 + b'"}]')
    assert 15_400_000 < body.size < 16_200_000
    want = oracle.parse(3, body, ARRAY)
    with pj.Context(device=0) as c:
        for _ in range(3):
            assert same_result(want, gpu_parse_device(c, 3, body, ARRAY)) == ""
