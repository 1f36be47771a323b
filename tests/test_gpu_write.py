"""k_write_tile on tables that its tiles are not made for, against the checker; the same on the CPU: test_write_emulation.py."""
import random

import numpy as np
import pytest

from pj_testlib import abi, as_u8, pj
from test_write_emulation import COL, MIXED, NDJSON, ARRAY, PET, USER, edge_text, fall, long_text

pytestmark = pytest.mark.gpu


def check(ctx, oracle, schema, cols, inclusion=abi.PJ_INCLUDE_NON_EMPTY, framings=(NDJSON, ARRAY)):
    """From device columns to device text at an odd address, and from host columns to host text."""
    import torch

    dev = pj.DeviceColumns.from_host(cols, "cuda")
    for framing in framings:
        want = oracle.write(schema, cols, framing, inclusion)
        out = torch.zeros(want.size + 80, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        for off in (0, 5):
            n = ctx.write(schema, dev, out[off:off + want.size], framing)
            assert n == want.size and np.array_equal(out[off:off + n].cpu().numpy(), want)
        assert not out[5 + want.size:].any()
        host = np.zeros(want.size, np.uint8)
        assert ctx.write(schema, cols, host, framing) == want.size and np.array_equal(host, want)


def users(n, size, esc):
    word = lambda i, k: "".join('\\"' if esc and (j + i) % esc == 3 else "q" for j in range(size + (i * 7 + k) % 5))
    return as_u8("\n".join('{"id":%d,"username":"%s","email":"%s","phone":"%s"}' % (i, word(i, 0), word(i, 1), word(i, 2)) for i in range(n)))


@pytest.mark.parametrize("esc", [0, 150])
@pytest.mark.parametrize("size", [511, 512, 2048, 5000, 9000, 30_000])
def test_long_strings(ctx, oracle, size, esc):
    """Staged with others, one to a window, and beyond what is staged."""
    check(ctx, oracle, USER, oracle.parse(USER, users(400 if size < 4000 else 40, size, esc)))


@pytest.mark.parametrize("size, esc", [(5, 2), (20, 7), (47, 3), (48, 3), (70, 60), (520, 9)])
def test_many_bytes_to_escape(ctx, oracle, size, esc):
    """Strings looked over one per lane; those shorter than 48 bytes escaped by the lanes that meet them."""
    check(ctx, oracle, USER, oracle.parse(USER, users(3000 if size < 500 else 300, size, esc)))
    line = '{"id":%d,"category":{"name":"%s"},"name":"%s","photoUrls":["%s",""],"tags":[{"name":"%s"}]}'
    text = lambda i: "".join('\\n' if (j + i) % esc == 1 else "p" for j in range(size))
    check(ctx, oracle, PET, oracle.parse(PET, as_u8("\n".join(line % (i, text(i), text(i + 1), text(i + 2), text(i + 3)) for i in range(1500 if size < 500 else 200)))))


@pytest.mark.parametrize("text", ['{"name":"","photoUrls":[]}', '{"id":%d,"name":"ab","photoUrls":[]}', '{"id":%d,"name":"say \\"%d\\"","photoUrls":["u","\\n"],"tags":[{"id":%d}],"status":"sold"}'])
def test_many_short_pets(ctx, oracle, text):
    """Tables of four blocks to an SM; and of few tiles, which are not."""
    for n in (150_001, 2000):
        check(ctx, oracle, PET, oracle.parse(PET, as_u8("\n".join(text.replace("%d", str(i)) for i in range(n)))))


@pytest.mark.parametrize("dirty", [0, 0.01])
def test_long_lists_and_records_of_all_sizes(ctx, oracle, dirty):
    rng = random.Random(3)
    cols = oracle.parse(PET, np.concatenate([long_text(rng, 60, dirty), as_u8(b"\n"), pj.gen_text(PET, 3, 0, 3000, abi.PJ_GEN_ZIPF_LISTS), long_text(rng, 5, dirty)]))
    assert cols.n_errors == 0
    check(ctx, oracle, PET, cols)
    cols = oracle.parse(PET, as_u8(b"\n".join(b'{"id":%d,"name":"n","photoUrls":[%s]}' % (i, b",".join(b'"%s"' % (b"u" * (60 + i % 3)) for _ in range(700 + 300 * (i % 5)))) for i in range(60))))
    check(ctx, oracle, PET, cols, framings=(NDJSON,))


@pytest.mark.parametrize("seed", range(3))
def test_rounds_of_a_window(ctx, oracle, seed):
    cols = oracle.parse(PET, edge_text(random.Random(seed), 700))
    assert cols.n_errors == 0
    check(ctx, oracle, PET, cols)


@pytest.mark.parametrize("flags", [0, abi.PJ_GEN_ESCAPES])
@pytest.mark.parametrize("how", ["reverse", "shuffle", "drop", "repeat"])
def test_records_in_the_callers_order(ctx, oracle, how, flags):
    cols = oracle.parse(MIXED, np.concatenate([pj.gen_text(MIXED, 9, 0, 4000, flags), long_text(random.Random(1), 8, 0.01 if flags else 0)]))
    n = cols.n_records
    kind, row = cols.arrays[COL["rec_type"]][:n], cols.arrays[COL["rec_row"]].view(np.uint32)[:n]
    if how == "drop":
        kind[::10] = abi.PJ_TYPE_NONE
    else:
        p = {"reverse": np.arange(n)[::-1], "shuffle": np.random.default_rng(2).permutation(n), "repeat": np.arange(n) // 3}[how]
        kind[:], row[:] = kind[p].copy(), row[p].copy()
    check(ctx, oracle, MIXED, cols)


def test_offsets_that_fall_where_no_string_is(ctx, oracle):
    cols = oracle.parse(USER, as_u8("\n".join('{"id":%d,"username":"%s","email":"%s"}' % (i, '\\"x\\n' * 4, "\\u0001y" * 5) for i in range(600))))
    for row in range(1, 599, 7):
        cols.arrays[COL["usr_present"]][row] &= ~2 & 0xFF
        fall(cols.arrays[COL["usr_username_off"]].view(np.uint32), row, 9)
    check(ctx, oracle, USER, cols)
