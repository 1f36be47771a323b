"""The work that users of petjson have it do, as cases whose time is measured.

A program that uses this library keeps one handle (a Context, as the mapper bean of a service) and passes text and
column buffers to it: it parses request bodies and exports into typed columns, writes columns back as JSON, or asks for
the record index alone. A case says which of these, on what records, in which framing, from where to where and with
which options. The value distributions are the workload generator's (petjson_gen.h), which are those of the benchmark
configurations; the text of a case depends on its seed alone.

    op         "parse" | "write" | "index"
    models     "pet" | "order" | "user" | "mixed"
    records    how many
    array      one JSON array instead of a record per line
    zipf       list lengths zipf(1.2): tags up to 64, photoUrls up to 256, instead of 0-3 and 0-4
    escapes    5 % of the strings hold escapes, surrogate pairs and UTF-8
    blanks     random blanks between the tokens (another producer's spelling)
    sparse     optional properties missing or null
    malformed  1 % of the records fail validation
    lenient    the handle is opened with the permissive answers of the rules (PJ_OPT_*)
    inclusion  "non_empty" | "non_null" | "always": which properties the writer writes
    memory     "device" | "host" | "pinned": where text and columns lie
    offset     device text starts that many bytes behind an aligned address (a slice of a larger buffer)
"""
import concurrent.futures
import functools
import importlib
import math
import os

import numpy as np
import torch

pj = importlib.import_module("micronaut3-bug_b200")
abi = pj.abi

SCHEMA = {"pet": abi.PJ_SCHEMA_PET, "order": abi.PJ_SCHEMA_ORDER, "user": abi.PJ_SCHEMA_USER, "mixed": abi.PJ_SCHEMA_MIXED}
INCLUSION = {"non_empty": abi.PJ_INCLUDE_NON_EMPTY, "non_null": abi.PJ_INCLUDE_NON_NULL, "always": abi.PJ_INCLUDE_ALWAYS}
TEXT_FLAGS = {"zipf": abi.PJ_GEN_ZIPF_LISTS, "escapes": abi.PJ_GEN_ESCAPES, "blanks": abi.PJ_GEN_WHITESPACE,
              "malformed": abi.PJ_GEN_MALFORMED, "array": abi.PJ_GEN_ARRAY, "sparse": abi.PJ_GEN_SPARSE}
LENIENT = abi.PJ_OPT_ENUM_UNKNOWN_AS_NULL | abi.PJ_OPT_LONE_SURROGATE_REPLACE | abi.PJ_OPT_COERCE_SCALARS
DEFAULTS = {"op": "parse", "models": "pet", "records": 1, "array": False, "zipf": False, "escapes": False, "blanks": False, "sparse": False,
            "malformed": False, "lenient": False, "inclusion": "non_null", "memory": "device", "offset": 0}
RECORD_BYTES = {"pet": 295, "order": 146, "user": 186, "mixed": 229}  # of text, short lists
ZIPF_FACTOR = {"pet": 6, "order": 1, "user": 1, "mixed": 4}           # times that with zipf lists


def _case(**kw):
    return {**DEFAULTS, **kw}


def listed():
    return [
        # one page of a REST list: a request body of the web tier, from host memory to host memory and back
        _case(name="page_read", records=20, array=True, memory="host"),
        _case(name="page_write", op="write", records=20, array=True, memory="host"),
        # the reference's own case: a JSON array of 1000 Pets
        _case(name="pets_array_1k", records=1000, array=True),
        # a batch of a message queue, a few thousand compact records
        _case(name="orders_5k", models="order", records=5000),
        # a partner's export: blanks, missing and null properties
        _case(name="users_200k_spaced", models="user", records=200_000, blanks=True, sparse=True),
        # a document export as one array, with escapes
        _case(name="pets_array_100k", records=100_003, array=True, escapes=True),
        # the benchmark configuration: 1 M Pets, one per line, resident on the GPU
        _case(name="pets_1m", records=1_000_000),
        # event stream of three models, 1 % broken
        _case(name="mixed_2m", models="mixed", records=2_000_000, malformed=True),
        # long lists, escapes and blanks
        _case(name="pets_zipf_100k", records=100_000, zipf=True, escapes=True, blanks=True),
        # the benchmark's end-to-end leg: pinned text in, every column back to pinned memory
        _case(name="pets_1m_pinned", records=1_000_000, memory="pinned"),
        # columns to text: the benchmark's reverse direction, and a mixed table with escapes and explicit nulls
        _case(name="pets_1m_write", op="write", records=1_000_000),
        _case(name="mixed_300k_write", op="write", models="mixed", records=300_001, escapes=True, sparse=True, inclusion="always"),
    ]


def draw(rng):
    op = rng.choice(["parse"] * 5 + ["write"] * 3 + ["index"])
    models = rng.choice(["pet", "pet", "order", "user", "mixed"])
    c = _case(op=op, models=models, array=rng.random() < 0.3, zipf=models in ("pet", "mixed") and rng.random() < 0.2,
              escapes=rng.random() < 0.35, blanks=op != "write" and rng.random() < 0.3, sparse=rng.random() < 0.35,
              malformed=op == "parse" and rng.random() < 0.3, inclusion=rng.choice(list(INCLUSION)))
    c["lenient"] = c["malformed"] and rng.random() < 0.3
    c["memory"] = "device" if op == "index" else rng.choice(["device"] * 3 + ["host", "pinned"])
    c["offset"] = rng.randrange(16) if c["memory"] == "device" and rng.random() < 0.4 else 0
    most = 300e6 if c["memory"] == "device" else 60e6
    if c["zipf"]:
        most = min(most, 20e6 if c["array"] else 120e6)
    per = RECORD_BYTES[models] * (ZIPF_FACTOR[models] if c["zipf"] else 1)
    c["records"] = max(1, round(math.exp(rng.uniform(math.log(per), math.log(most))) / per))
    return c


# ---- inputs ---------------------------------------------------------------------------------------------
def _text(case, seed, n):
    """JSON text of the case's first n records, made by all cores side by side."""
    schema, array = SCHEMA[case["models"]], case["array"]
    flags = sum(v for k, v in TEXT_FLAGS.items() if case[k])
    room = 4000 if case["zipf"] else 1000

    def part(first, count):
        try:
            t = pj.gen_text(schema, seed, first, count, flags, out=np.empty(count * room + 800_000, np.uint8))
        except pj.PetJsonError:  # unusually long records
            t = pj.gen_text(schema, seed, first, count, flags)
        return t[1:-1] if array else t

    part(0, 1)  # the generator's tables are set up by its first call
    step = max(2000, -(-n // (2 * (os.cpu_count() or 1))))
    with concurrent.futures.ThreadPoolExecutor() as pool:
        parts = list(pool.map(lambda first: part(first, min(step, n - first)), range(0, n, step)))
    if array:
        out = [np.frombuffer(b"[", np.uint8)]
        for p in parts:
            out += [p, np.frombuffer(b",", np.uint8)]
        out[-1] = np.frombuffer(b"]", np.uint8)
        parts = out
    return np.concatenate(parts)


def _items(case):
    """List elements of a kind that the case's records can hold (zipf lists: 27 photoUrls a record on average, up to 256)."""
    n = case["records"] + 1
    return 40 * n + 500 * math.isqrt(n) if case["zipf"] else 4 * n


def _caps(case):
    """Bytes per column buffer: what a program that knows its data allocates (strings below 40 bytes, photoUrls below 80)."""
    n, items = case["records"] + 1, _items(case) + 1
    caps = {}
    for c in abi.schema_columns(SCHEMA[case["models"]]):
        if c.shape == "bytes":
            caps[c.id] = {"pet_photo_data": 80 * items, "pet_tag_name_data": 40 * items}.get(c.name, 40 * n)
        else:
            caps[c.id] = (n if c.shape in ("rows", "rows+1") else items) * np.dtype(c.dtype).itemsize
    return caps


def _pinned(nbytes):
    return torch.zeros(nbytes, dtype=torch.uint8, pin_memory=True).numpy()


@functools.cache
def _handle(inclusion, flags):
    """The program's one handle per set of options, kept for its whole life."""
    return pj.Context(device=0, inclusion=inclusion, flags=flags)


def _columns(case):
    schema, caps = SCHEMA[case["models"]], _caps(case)
    if case["memory"] == "device":
        cols = pj.DeviceColumns(schema, caps, "cuda:0")
        for t in cols.tensors.values():
            t.zero_()
        return cols
    return abi.HostColumns(schema, caps, alloc=_pinned if case["memory"] == "pinned" else None)


def _place(case, text):
    if case["memory"] == "host":
        return text
    if case["memory"] == "pinned":
        buf = _pinned(text.size)
        buf[:] = text
        return buf
    buf = torch.empty(text.size + 16, dtype=torch.uint8, device="cuda:0")[case["offset"]:][: text.size]
    buf.copy_(torch.from_numpy(text))
    return buf


def prepare(case, seed):
    case = {**DEFAULTS, **case}
    framing = abi.PJ_FRAMING_ARRAY if case["array"] else abi.PJ_FRAMING_NDJSON
    state = {"op": case["op"], "schema": SCHEMA[case["models"]], "framing": framing,
             "ctx": _handle(INCLUSION[case["inclusion"]], LENIENT if case["lenient"] else 0)}
    text = _text(case, seed, case["records"])
    if case["op"] == "index":
        state["text"] = _place(case, text)
        state["starts"] = torch.zeros(case["records"] + 1, dtype=torch.int64, device="cuda:0")
        return state
    cols = state["cols"] = _columns(case)
    buffers = cols.tensors if case["memory"] == "device" else cols.arrays
    if case["op"] == "parse":
        state["text"] = _place(case, text)
        state["columns"] = {c.name: buffers[c.id] for c in abi.schema_columns(state["schema"])}
    else:  # the table to write: what parsing the text gave
        torch.cuda.synchronize()
        state["ctx"].parse(state["schema"], _place(case, text), cols, framing)
        room = 800 * case["records"] + (80 * _items(case) if case["zipf"] else 0) + 4096
        if case["memory"] == "device":
            state["out"] = torch.zeros(room, dtype=torch.uint8, device="cuda:0")
        else:
            state["out"] = _pinned(room) if case["memory"] == "pinned" else np.zeros(room, np.uint8)
    torch.cuda.synchronize()
    return state


def run(state):
    if state["op"] == "parse":
        cols = state["cols"]
        state["ctx"].parse(state["schema"], state["text"], cols, state["framing"])
        return {"columns": state["columns"], "records": cols.n_records, "errors": cols.n_errors, "rows": [cols.n_rows(t) for t in (1, 2, 3)]}
    if state["op"] == "write":
        return {"bytes": state["ctx"].write(state["schema"], state["cols"], state["out"], state["framing"]), "text": state["out"]}
    return {"records": state["ctx"].index_records(state["text"], state["starts"], state["framing"]), "starts": state["starts"]}


# ---- what a pass cannot do without ----------------------------------------------------------------------
@functools.cache
def _per_record(models, flags):
    """(text bytes, column bytes without the record columns, record column bytes) per record, from a sample of the records."""
    schema, n = SCHEMA[models], 3000
    text = pj.gen_text(schema, 1, 0, n, flags).size
    cols = pj.gen_columns(schema, 1, 0, n, flags, text)
    size = {c.name: cols.count(c.id) * np.dtype(c.dtype).itemsize for c in abi.schema_columns(schema)}
    own = sum(size[c.name] for c in abi.schema_columns(schema) if c.owner == 0)
    return text / n, (sum(size.values()) - own) / n, own / n


def work(case):
    case = {**DEFAULTS, **case}
    text, table, own = _per_record(case["models"], sum(v for k, v in TEXT_FLAGS.items() if case[k] and k != "array"))
    per = {"parse": text + table + own, "write": table + text, "index": text + 8}[case["op"]]
    return {"bytes": per * case["records"], "flops": 0}


def tolerance(case):
    return "exact"  # integers and bytes
