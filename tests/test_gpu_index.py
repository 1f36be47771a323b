"""The record index, the separators of arrays and the small calls' way back, at the sizes where another variant takes over, against the checker."""
import numpy as np
import pytest

from pj_testlib import abi, as_u8, pj, same_result
from test_gpu_parity import ARRAY, NDJSON, gpu_parse_device, gpu_parse_host

pytestmark = pytest.mark.gpu

PET, ORDER, MIXED = abi.PJ_SCHEMA_PET, abi.PJ_SCHEMA_ORDER, abi.PJ_SCHEMA_MIXED


def four_words():
    """Bytes from which a thread of the index takes four words instead of one."""
    import torch

    return torch.cuda.get_device_properties(0).multi_processor_count * 2 * 64 * 1024


def text_of(size, array):
    """`size` bytes of Pets with blanks and escapes; line feeds or commas on and beside the edges of words and tiles."""
    sep = b"," if array else b"\n"
    lines = bytes(pj.gen_text(PET, 77, 0, size // 300 + 2000, abi.PJ_GEN_ESCAPES | abi.PJ_GEN_WHITESPACE)).split(b"\n")
    out, at, k = [b"[" if array else b""], int(array), 0
    for line in lines:
        edge = (at + len(line)) // 16_384 * 16_384 + 16_383 + k % 3  # the separator goes there, if this is the last record before it
        pad = edge - at - len(line) if 0 <= edge - at - len(line) < 400 else 0
        k += pad > 0
        if at + len(line) + pad + 500 > size:
            break
        out.append(line + b" " * pad + sep)
        at += len(line) + pad + 1
    return as_u8(b"".join(out) + b'{"id":1}' + b" " * (size - at - 9) + (b"]" if array else b"\n"))


@pytest.mark.parametrize("framing", [NDJSON, ARRAY])
@pytest.mark.parametrize("mb", [-1, 1, 6])
def test_record_index_around_four_words(ctx, oracle, framing, mb):
    import torch

    size = four_words() + mb * 1_000_000
    body = text_of(size, framing == ARRAY)
    want = oracle.index(body, framing)
    assert want.size > 1000
    for off in (0, 1, 15):
        buf = torch.empty(size + 64, dtype=torch.uint8, device="cuda")[off:off + size]
        buf.copy_(torch.from_numpy(body))
        starts = torch.zeros(want.size + 1, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        assert ctx.index_records(buf, starts, framing) == want.size
        got = starts.cpu().numpy().view(np.uint64)
        assert np.array_equal(got[:-1], want) and got[-1] == 0
    assert ctx.index_records(buf, starts[:10], framing, allow_capacity=True) == want.size


@pytest.mark.parametrize("mb", [-1, 1, 6])
def test_arrays_around_four_words(ctx, oracle, mb):
    size = four_words() + mb * 1_000_000
    body = pj.gen_text(PET, 78, 0, size // 290 + 2000, abi.PJ_GEN_ARRAY | abi.PJ_GEN_ESCAPES)[:size].copy()
    end = body.size - 1 - int(np.argmax(body[::-1] == ord("}")))
    body[end + 1:] = ord(" ")
    body[-1] = ord("]")  # a last record that may be cut short
    want = oracle.parse(PET, body, ARRAY)
    for off in (0, 1, 15):
        assert same_result(want, gpu_parse_device(ctx, PET, body, ARRAY, off)) == ""


@pytest.mark.parametrize("framing", [NDJSON, ARRAY])
def test_calls_of_16_mb(ctx, oracle, framing):
    """Up to 16 MB a call's result comes by a kernel, beyond by a copy."""
    base = pj.gen_text(ORDER, 5, 0, 100_000, abi.PJ_GEN_ARRAY if framing == ARRAY else 0)
    want = oracle.parse(ORDER, base, framing)
    for size in ((16 << 20) - 1, 16 << 20, (16 << 20) + 1):
        body = np.full(size, ord(" "), np.uint8)
        body[:base.size] = base
        assert same_result(want, gpu_parse_device(ctx, ORDER, body, framing)) == "", size
        assert same_result(want, gpu_parse_host(ctx, ORDER, body, framing)) == "", size


def column_bytes(cols):
    """Of the columns of a result, each rounded up as it lies in the buffer it is fetched through."""
    return sum((cols.count(c.id) * np.dtype(c.dtype).itemsize + 15) // 16 * 16 for c in abi.schema_columns(cols.schema))


def test_columns_around_the_room_they_come_back_through(ctx, oracle):
    """1 MB of columns comes back with the result, more by copies."""
    line = b'{"id":12345,"petId":7,"quantity":1}'
    per = column_bytes(oracle.parse(ORDER, as_u8(b"\n".join([line] * 4000)))) / 4000
    near = int((1 << 20) / per)
    seen = set()
    for n in [1, near // 2, *range(near - 4, near + 5), near + 300]:
        for framing, body in ((NDJSON, b"\n".join([line] * n)), (ARRAY, b"[" + b",".join([line] * n) + b"]")):
            assert len(body) <= 786_432
            want = oracle.parse(ORDER, as_u8(body), framing)
            seen.add(column_bytes(want) > 1 << 20)
            assert same_result(want, gpu_parse_host(ctx, ORDER, body, framing)) == "", n
    assert seen == {False, True}
    for size in (786_432 - 1, 786_432, 786_432 + 1):  # the input size up to which they are tried
        body = line + b"\n" + line + b" " * (size - 2 * len(line) - 1)
        assert same_result(oracle.parse(ORDER, as_u8(body)), gpu_parse_host(ctx, ORDER, body)) == ""


@pytest.mark.parametrize("framing", [NDJSON, ARRAY])
def test_text_around_the_room_it_comes_back_through(ctx, oracle, framing):
    text = pj.gen_text(ORDER, 6, 0, 24_000, 0)
    ends = np.flatnonzero(text == 10) + 1
    near = int(np.searchsorted(ends, 1 << 20))
    seen = set()
    for n in [1, 2000, *range(near - 3, near + 4), near + 400, 24_000]:  # (the last ones: more columns than one copy takes)
        cols = oracle.parse(ORDER, text[:ends[n - 1]])
        want = oracle.write(ORDER, cols, framing, abi.PJ_INCLUDE_NON_EMPTY)
        out = np.zeros(want.size + 8, np.uint8)
        assert ctx.write(ORDER, cols, out, framing) == want.size and np.array_equal(out[:want.size], want) and not out[want.size:].any(), n
        seen.add(want.size > 1 << 20)
    assert seen == {False, True}


@pytest.mark.parametrize("what", ["array", "index", "index array", "write", "write array"])
def test_a_bounded_wait_that_runs_out(native, oracle, what):
    """Tile 0 of the first call is never handed out (test hook): PJ_ERR_TIMEOUT after 2 ms, and the same context answers the next call."""
    import torch

    framing = ARRAY if "array" in what else NDJSON
    text = pj.gen_text(PET, 8, 0, 20_000, abi.PJ_GEN_ARRAY if framing == ARRAY else 0)
    cols = oracle.parse(PET, text, framing)
    with native.Context(device=0, flags=abi.PJ_OPT_TEST_STALL_ONCE, spin_limit_us=2000) as c:
        if "write" in what:
            want = oracle.write(PET, cols, framing, abi.PJ_INCLUDE_NON_EMPTY)
            dev = pj.DeviceColumns.from_host(cols, "cuda")
            out = torch.zeros(want.size, dtype=torch.uint8, device="cuda")
            call = lambda: c.write(PET, dev, out, framing) == want.size and np.array_equal(out.cpu().numpy(), want)
        elif "index" in what:
            want = oracle.index(text, framing)
            buf, starts = torch.from_numpy(text).cuda(), torch.zeros(want.size, dtype=torch.int64, device="cuda")
            call = lambda: c.index_records(buf, starts, framing) == want.size and np.array_equal(starts.cpu().numpy().view(np.uint64), want)
        else:
            call = lambda: same_result(cols, gpu_parse_device(c, PET, text, framing)) == ""
        torch.cuda.synchronize()
        with pytest.raises(native.PetJsonError) as e:
            call()
        assert e.value.status == abi.PJ_ERR_TIMEOUT
        assert call() and call()


@pytest.mark.parametrize("edge", [8 << 20, 64 << 20])
def test_record_index_where_the_input_is_read_twice(ctx, oracle, edge):
    """Between 8 and 64 MB two passes, else one."""
    import torch

    body = text_of(edge + 1, False)
    buf = torch.empty(body.size + 16, dtype=torch.uint8, device="cuda")
    for size in (edge - 1, edge, edge + 1):
        want = oracle.index(body[:size], NDJSON)
        for off in (0, 5):
            buf[off:off + size].copy_(torch.from_numpy(body[:size]))
            starts = torch.zeros(want.size + 1, dtype=torch.int64, device="cuda")
            torch.cuda.synchronize()
            assert ctx.index_records(buf[off:off + size], starts, NDJSON) == want.size
            got = starts.cpu().numpy().view(np.uint64)
            assert np.array_equal(got[:-1], want) and got[-1] == 0
        assert ctx.index_records(buf[5:5 + size], starts[:10], NDJSON, allow_capacity=True) == want.size
