"""What may begin before the launch ahead has finished (csrc/tq_stream_order.h), stepped through on the CPU for every
sequence of the library's launches on a stream, with other streams' notes taking the place of this one's anywhere between.

The model of a launch follows the places that launch it: whether it is a programmatic dependent, whether it lets its own
dependents begin at entry, after its wait or only by finishing, what it writes, and whether it reads the pool or rows in front of
its wait.  What a launch wrote is there for an early reader only if some launch in between has waited for it.
"""

import ctypes as C
import itertools
import os
import re
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "turboquant_b200", "csrc")
UNKNOWN, DECODE, STORE_EARLY, NEUTRAL, PREP_BEHIND_STORE, WAITED, STORE_PLAIN = range(7)
GLUE = """
#include "tq_stream_order.h"
extern "C" {
int kind_of_prep(int k) { return tq_kind_of_prep(k); }
int may_overlap(int k) { return tq_reader_may_overlap(k); }
int pool_is_late(int k) { return tq_pool_is_late(k); }
int rows_at_rest(int k) { return tq_rows_are_at_rest(k); }
void* notes_new() { return new TqStreamNotes; }
void notes_free(void* n) { delete static_cast<TqStreamNotes*>(n); }
void note(void* n, unsigned long st, int k) { static_cast<TqStreamNotes*>(n)->note(reinterpret_cast<const void*>(st), k); }
int last(void* n, unsigned long st) { return static_cast<TqStreamNotes*>(n)->last(reinterpret_cast<const void*>(st)); }
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("stream_order")
    (d / "glue.cpp").write_text(GLUE)
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, "-o", str(d / "glue.so"), str(d / "glue.cpp")],
                   check=True)
    lib = C.CDLL(str(d / "glue.so"))
    lib.notes_new.restype = C.c_void_p
    lib.notes_free.argtypes = [C.c_void_p]
    lib.note.argtypes = [C.c_void_p, C.c_ulong, C.c_int]
    lib.last.argtypes = [C.c_void_p, C.c_ulong]
    return lib


def _launch(r, name, ahead):
    """(programmatic, lets others begin, writes, reads early, note or None) of a launch behind one noted as `ahead`."""
    if name == "store":
        late = not r.rows_at_rest(ahead)
        return True, "waited" if late else "entry", "pool", None if late else "rows", STORE_EARLY
    if name == "fp32 store":                  # and planes into the pool
        return False, "done", "pool", None, STORE_PLAIN
    if name == "ring write":
        return True, "waited", "rows", None, DECODE
    if name == "prepare":                     # may append a row to the ring
        return True, "entry", "rows", None, r.kind_of_prep(ahead)
    if name == "decode":
        prog, late = bool(r.may_overlap(ahead)), bool(r.pool_is_late(ahead))
        return prog, "waited" if late else "entry", None, "pool" if prog and not late else None, DECODE
    if name == "cache scores":
        return True, "done", None, None if r.pool_is_late(ahead) else "pool", None
    if name == "cache attend":
        return True, "done", None, None, WAITED
    if name == "plain rows":
        return True, "waited", "rows", None, WAITED
    assert name == "prefill"
    return False, "entry", None, None, NEUTRAL


LAUNCHES = ("store", "fp32 store", "ring write", "prepare", "decode", "cache scores", "cache attend", "plain rows", "prefill")


def _run(r, steps):
    """None, or what went wrong."""
    notes, loose = r.notes_new(), set()
    try:
        for name in steps:
            if name == "others":              # eight other streams launch something
                for st in range(100, 108):
                    r.note(notes, st, DECODE)
                continue
            prog, begin, writes, early, kind = _launch(r, name, r.last(notes, 7))
            if prog and early in loose:
                return "%s reads %s that may not be written" % (name, early)
            loose = (loose if prog and begin == "entry" else set()) | ({writes} if writes else set())
            if kind is not None:
                r.note(notes, 7, kind)
    finally:
        r.notes_free(notes)
    return None


def test_nobody_reads_early_what_may_not_be_written(rules):
    wrong = []
    for n in range(1, 6):
        for steps in itertools.product(LAUNCHES + ("others",), repeat=n):
            bad = _run(rules, steps)
            if bad:
                wrong.append((steps, bad))
                if len(wrong) > 3:
                    break
    assert not wrong, wrong


@pytest.mark.parametrize("reader", ["decode", "cache scores"])
def test_readers_overlap_where_the_pool_is_known_to_be_at_rest(rules, reader):
    """The usual steps keep their early reads: behind another step, a ring write, attention of the cache object or a prefill."""
    for ahead in (DECODE, NEUTRAL, WAITED):
        kind = rules.kind_of_prep(ahead)
        assert kind == DECODE and _launch(rules, reader, kind)[3] == "pool"
    assert all(rules.rows_at_rest(k) for k in (STORE_EARLY, NEUTRAL, STORE_PLAIN))


def test_notes_keep_the_last_eight_streams(rules):
    notes = rules.notes_new()
    for st in range(1, 9):
        rules.note(notes, st, STORE_EARLY)
    rules.note(notes, 3, DECODE)
    assert [rules.last(notes, st) for st in (1, 3, 8)] == [STORE_EARLY, DECODE, STORE_EARLY]
    rules.note(notes, 9, NEUTRAL)
    assert rules.last(notes, 1) == UNKNOWN and rules.last(notes, 9) == NEUTRAL and rules.last(notes, 2) == STORE_EARLY
    rules.notes_free(notes)


@pytest.mark.parametrize("kernel,begin,first_use", [
    ("tq_store_tc_kernel", "in the order they are needed", "if (rmw)"),                  # loads and products
    ("tq_store_tc_kernel", "compute warps ====", "bool ok = phase_n_and_arrive(0"),
    ("tq_store_tc256_kernel", "if (warp == TC_THREADS / 32) {\n", "wait1(bar_n"),         # products
    ("tq_store_tc256_kernel", "int loaded = 0;", "issue_rows(sA0"),                       # loads; the operands' first boxes wait for nobody
    ("tq_store_tc256_kernel", "compute warps ====", "const int64_t tok0 = tile_tok0(tile);"),
])
def test_every_warp_of_a_late_store_waits_for_the_launch_ahead_first(kernel, begin, first_use):
    """The waits on barriers are bounded, and their bound is meant for the kernel's own phases: behind a launch that may be
    writing rows no warp of a store polls a barrier before it has waited for that launch.  Read from the source, role by role."""
    text = open(os.path.join(CSRC, "tq_store_tc.cu")).read()
    body = text[text.index(kernel + "("):]
    body = body[body.index("issuing"):]
    body = body[body.index(begin):]
    body = body[:body.index(first_use)]
    assert re.search(r"if \(p\.rows_late\)[\s{].*(pool_writes_may_begin|rows_may_be_read)\(\)", body, re.S), body


def test_no_read_only_loads_of_what_the_launch_ahead_may_write():
    """A grid that is resident while the launch ahead still writes must not read that through pointers which promise the compiler
    that nobody does (`const ... __restrict__`: such loads may move in front of the wait).  Constant operands are written once,
    before any launch; the staging kernel's source is host memory."""
    constants = {"pi", "s", "pi_t", "s_t"}
    seen, wrong = 0, []
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith(".cu"):
            continue
        text = open(os.path.join(CSRC, name)).read()
        starts = [m.start() for m in re.finditer(r"__global__ void", text)] + [len(text)]
        for a, b in zip(starts, starts[1:]):
            kernel, args = re.match(r"__global__ void (?:__launch_bounds__\([^)]*\)\s*)?(\w+)\((.*?)\) \{", text[a:b], re.S).groups()
            if not re.search(r"griddepcontrol\.wait|wait_for_launch_ahead\(\)|pool_writes_may_begin\(\)", text[a:b]):
                continue
            seen += 1
            for ptr in re.findall(r"const \w+\* __restrict__ (\w+)", args):
                if ptr not in constants and kernel != "tq_stage_in_kernel":
                    wrong.append((kernel, ptr))
    assert seen >= 12 and not wrong, (seen, wrong)
