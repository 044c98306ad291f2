"""The host side of the attention library over a CUDA runtime that only keeps a record: what is drawn, kept and given back."""
import ctypes as C
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("g++ not available")
    so = str(tmp_path_factory.mktemp("fa") / "libfa_fake.so")
    cmd = ["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", os.path.join(CUDA, "include"), "-x", "c++",
           *(os.path.join(ROOT, "goml_b200", "csrc", f) for f in ("fa_api.cu", "fa_dispatch.cpp")), os.path.join(ROOT, "tests", "host_cpp", "fake_runtime.cpp"), "-o", so, "-lpthread"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = C.CDLL(so)
    lib.fake_log.restype = C.c_char_p
    lib.fa_create.argtypes = [C.POINTER(C.c_void_p)]
    lib.fa_destroy.argtypes = [C.c_void_p]
    lib.fa_forward.argtypes = [C.c_void_p] * 5 + [C.c_int] * 5 + [C.c_float, C.c_void_p]
    return lib


class Context:
    def __init__(self, lib):
        self.lib, self.ptr = lib, C.c_void_p()
        assert lib.fa_create(C.byref(self.ptr)) == 0

    def forward(self, stream, bh=4, ok=True):
        """One call on a stream (its handle is its id); the lines it left in the record."""
        self.lib.fake_clear()
        assert (self.lib.fa_forward(self.ptr, 0x10, 0x10, 0x10, 0x10, bh, 256, 64, 0, 0, 0.1, stream) == 0) == ok
        return self.lib.fake_log().decode().splitlines()

    def destroy(self):
        self.lib.fake_clear()
        self.lib.fa_destroy(self.ptr)
        return self.lib.fake_log().decode().splitlines()


def field(lines, what, name):
    return [re.search(rf"\b{name} (\d+)", x).group(1) for x in lines if x.startswith(what)]


def test_the_last_context_gives_back_without_waiting(library):
    # every kept buffer is freed on a stream of the library's own, behind the event recorded behind its stream's last call:
    # no synchronising call, which would stop the host and break a capture some other thread has begun
    a, b = Context(library), Context(library)
    kept, event = {}, {}
    for stream in (1, 2):
        for bh in (4, 400):    # the second call makes both buffers grow
            lines = (a if stream == 1 else b).forward(stream, bh)
            assert lines.index(next(x for x in lines if x.startswith("launch"))) < lines.index(next(x for x in lines if x.startswith("record")))
        kept[stream] = field(lines, "launch", "scratch") + field(lines, "launch", "flags")
        event[stream] = field(lines, "record", "event")
    assert a.destroy() == []   # the other context's calls go on
    lines = b.destroy()
    assert not [x for x in lines if x.startswith("SYNC")]
    for stream in (1, 2):
        for buf in kept[stream]:
            at = next(i for i, x in enumerate(lines) if x.startswith(f"free {buf} "))
            own = field([lines[at]], "free", "stream")[0]
            assert int(own) > 0x1000
            assert any(x == f"wait stream {own} event {event[stream][0]}" for x in lines[:at])
    assert len([x for x in lines if x.startswith("free")]) == 4 and [x.split()[0] for x in lines[-2:]] == ["pool_destroy", "stream_destroy"]


def test_what_a_failed_call_has_queued_is_covered_too(library):
    # the flags are drawn and cleared, the scratch is not to be had: the event stands behind the clearing
    ctx = Context(library)
    library.fake_fail_allocation(2)
    lines = ctx.forward(7, ok=False)
    assert [x.split()[0] for x in lines] == ["alloc", "memset", "record"]
    ctx.destroy()


def kept(lines):
    """Whether a call used buffers that it did not draw."""
    return not [x for x in lines if x.startswith("alloc")]


def test_streams_that_are_gone_give_their_place_up(library):
    # a stream per request: each finds a place again, and what it displaces is freed behind the displaced stream's last call
    ctx = Context(library)
    event = {}
    for stream in range(1, 9):
        event[stream] = field(ctx.forward(stream), "record", "event")[0]
    lines = ctx.forward(9)
    assert not field(lines, "record", "event") and not [x for x in lines if x.startswith("wait")]   # all places are in use
    for _ in range(70):
        assert kept(ctx.forward(8))
    lines = ctx.forward(10)           # in the place of stream 1
    freed = [x for x in lines if x.startswith("free")]
    assert len(freed) == 2 and lines.index(next(x for x in lines if x.startswith("wait"))) < lines.index(freed[0])
    assert field(lines, "wait", "event") == [event[1]] and not set(field(freed, "free", "stream")) & {str(s) for s in range(1, 11)}
    assert kept(ctx.forward(10)) and kept(ctx.forward(8))
    lines = ctx.forward(1)            # stream 1 is a new one again, in the place of stream 2
    assert field(lines, "wait", "event") == [event[2]] and kept(ctx.forward(1))
    ctx.destroy()


def test_more_streams_than_places_in_turn(library):
    # ten streams that call in turn: eight keep their buffers, two draw theirs for each call, nobody is displaced
    ctx = Context(library)
    for turn in range(30):
        for stream in range(1, 11):
            lines = ctx.forward(stream)
            assert not [x for x in lines if x.startswith("wait")]
            if turn:
                assert kept(lines) == (stream <= 8)
            if stream > 8:
                assert len([x for x in lines if x.startswith("free")]) == len([x for x in lines if x.startswith("alloc")]) == 1
    ctx.destroy()


def test_calls_without_scratch_leave_no_trace(library):
    # nothing drawn, kept, cleared or recorded; calls with scratch on the same stream go on as they were
    ctx = Context(library)
    ctx.forward(3)
    library.fake_rows_with_scratch(1000)
    try:
        for stream in (3, 4):
            assert ctx.forward(stream) == [f"launch stream {stream} scratch 0 flags 0"]
    finally:
        library.fake_rows_with_scratch(0)
    assert kept(ctx.forward(3)) and not kept(ctx.forward(4))
    ctx.destroy()
