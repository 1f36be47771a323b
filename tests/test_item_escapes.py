"""Strings with escapes and UTF-8 in k_parse_items, decoded by a thread each, four bytes a step: every kind of character at every place in a word and around
the 32nd and 64th byte, whole and broken, against the checker (on the CPU: tests/host_emu)."""
import random

import pytest

from pj_testlib import as_u8, same_result
from test_item_emulation import ARRAY, NDJSON, PET, USER, Run, emu  # noqa: F401 (emu: fixture)

GOOD = [b"\\n", b"\\\"", b"\\\\", b"\\/", b"\\u0041", b"\\u00e9", b"\\u20AC", b"\\ud83d\\ude00", b"\xc3\xa9", b"\xe2\x82\xac", b"\xf0\x9f\x98\x80", b"\xed\x9f\xbf", b"\xee\x80\x80", b"\xf4\x8f\xbf\xbf"]
BAD = [b"\\x", b"\\u12", b"\\u12g4", b"\\ud83d", b"\\ude00", b"\\ud83d\\n", b"\\ud83d\\ud83d\\ude00", b"\\ud83dx", b"\\ude00\\ud83d", b"\\ud83d\\u12", b"\\ud83d\\uzz00", b"\x01", b"\t", b"\x80", b"\xc3", b"\xc3x",
       b"\xe2\x82", b"\xe2\x82x", b"\xf0\x9f\x98", b"\xc0\x80", b"\xe0\x80\x80", b"\xed\xa0\x80", b"\xf4\x90\x80\x80", b"\xf5\x80\x80\x80", b"\xc3\xa9\xa9", b"\\u00\\n12"]


def user(i, s):
    return b'{"id":%d,"username":"%s","email":"%s"}' % (i, s, s[::1])


@pytest.mark.parametrize("opts", [0, 2])
@pytest.mark.parametrize("piece", GOOD + BAD, ids=lambda b: b.hex())
def test_every_place_around_a_step(emu, oracle, piece, opts):
    lines = []
    for lead in list(range(19, 34)) + [60, 63, 64]:
        for tail in (0, 1, 5, 40):
            lines.append(user(lead, b"a" * lead + piece + b"z" * tail))
    for k in range(0, len(lines), 30):  # few enough for a warp each
        body = as_u8(b"\n".join(lines[k:k + 30]))
        assert same_result(oracle.parse(USER, body, opts=opts), Run(emu, USER, body, opts=opts).cols) == "", k


def test_runs_of_pieces(emu, oracle):
    rng = random.Random(31)
    for it in range(60):
        lines = []
        for i in range(rng.choice([1, 8, 40, 90])):
            s = b"".join(rng.choice(GOOD if rng.random() < 0.97 else BAD) if rng.random() < 0.5 else b"x" * rng.randrange(9) for _ in range(rng.randrange(30)))
            t = b"".join(rng.choice(GOOD) for _ in range(rng.randrange(4)))
            lines.append(b'{"id":%d,"category":{"id":2,"name":"%s"},"name":"%s","photoUrls":["%s","b","%s"],"tags":[{"id":1,"name":"%s"},{"id":3,"name":"y"}],"status":"sold"}' % (i, s, t, s, t, s))
        opts = rng.choice([0, 2])
        framing = rng.choice([NDJSON, ARRAY])
        body = as_u8(b"\n".join(lines) if framing == NDJSON else b"[" + b",".join(lines) + b"]")
        got = Run(emu, PET, body, framing, opts=opts, order=it % 5)
        assert same_result(oracle.parse(PET, body, framing, opts=opts), got.cols) == "", it


def test_long_strings(emu, oracle):
    """More than 255 bytes freed, more strings of the kind than a warp each takes, spellings of names and literals."""
    body = as_u8(b"\n".join([user(1, b"\\u0041" * 300 + b"\xc3\xa9" * 200), user(2, b"\\n" * 999), b'{"\\u0069d":4,"username":"\\u0041"}', b'{"id":4,"username":"\\u0041","email":null}'] * 3))
    assert same_result(oracle.parse(USER, body), Run(emu, USER, body).cols) == ""
    body = as_u8(b"\n".join(user(i, b"\\u00e9" * (i % 7) + b"\xd0\x96") for i in range(250)))
    assert same_result(oracle.parse(USER, body), Run(emu, USER, body, str_words=8000).cols) == ""
    body = as_u8(b"\n".join(b'{"name":"\\u0041%d","photoUrls":[],"status":"%s"}' % (i, s) for i, s in enumerate([b"so\\u006cd", b"s\\u006fle", b"\\u0070ending", b"sold\\u0000"])))
    assert same_result(oracle.parse(PET, body), Run(emu, PET, body).cols) == ""
