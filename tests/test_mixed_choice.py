"""Which kernel streams of several models take (csrc/pj_choice.h): k_parse_items, unless a timed call of its like was slower with it."""
import ctypes as C
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def note(tmp_path_factory):
    lib = str(tmp_path_factory.mktemp("choice") / "libchoice.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I", os.path.join(os.path.dirname(HERE), "micronaut3-bug_b200", "csrc"), os.path.join(HERE, "host_emu", "pj_choice_emu.cpp"),
                    "-o", lib], check=True)
    cdll = C.CDLL(lib)

    def call(ms, records=100_000, per=200, fast=1.0, dense=1.0):
        return bool(cdll.mixed_choice_note(C.c_uint64(records * per), C.c_float(ms), C.c_uint64(records), C.c_uint64(int(records * fast)), C.c_uint64(int(records * dense))))

    call.reset = cdll.mixed_choice_reset
    return call


def test_compact_and_spaced_text_stay(note):
    note.reset()
    assert all(note(0.1, dense=d) for d in (1.0, 1.0, 0.0, 0.0, 1.0, 1.0, 1.0))
    assert all(note(0.05, records=n) for n in (10, 100, 1000, 5))


@pytest.mark.parametrize("stream_ms, ends", [(0.05, False), (0.5, True)])
def test_text_for_the_exact_parser_has_the_other_kernel_tried_once(note, stream_ms, ends):
    note.reset()
    took, items = [], True
    for _ in range(12):
        items = note(0.2 if items else stream_ms, fast=0.5)
        took.append(items)
    assert took[0] is False and all(t is ends for t in took[1:]), took


def test_small_calls_are_not_tried_in_turn(note):
    note.reset()
    assert all(note(0.02, records=500, fast=0.5) for _ in range(6))


def test_records_of_16_kb(note):
    note.reset()
    assert note(1.0, records=100, per=40_000) is False
    assert note(0.1, records=100, per=40_000) is False
    assert note(0.1) is True  # records of a usual size: back again


def test_long_records_between_usual_ones(note):
    """Calls of both kinds and of like size in turn: long records say nothing of what the kernels take for usual ones."""
    note.reset()
    items, seen = True, []
    for k in range(60):
        seen.append(items)
        if k % 3 == 0:  # 300 records of 40 KB
            items = note(15.6 if items else 0.5, records=300, per=40_000)
        else:           # 20 MB of usual ones
            items = note(0.25 if items else 0.31)
    assert all(seen[k] for k in range(60) if k % 3 == 2), seen
