"""libk2j's host side without a GPU: a child process runs it on a CUDA runtime of host memory (tests/native/fake_cudart.cpp)
whose allocations can be made to fail and whose kernels are noted and not run."""
import os
import shutil
import subprocess
import sys
import textwrap

import pytest

import helpers

pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")

PRELUDE = """
import ctypes as C, os, sys
import numpy as np
from kineto_b200 import api
fake = C.CDLL(os.environ["LD_PRELOAD"])
fake.fake_most.argtypes = [C.c_size_t]
fake.fake_pool_total.argtypes = fake.fake_scan_total.argtypes = [C.c_uint64]
OK, CUDA = 0, 2
lib = api.load_library()
ctx = C.c_void_p()
assert lib.k2j_create(0, None, C.byref(ctx)) == OK
params = api.Params()
assert lib.k2j_set_params(ctx, C.byref(params), None) == OK

def log():
    text = C.create_string_buffer(1 << 16)
    assert fake.fake_log(text, len(text)) >= 0
    return [l.split() for l in text.value.decode().splitlines()]

def rooms():  # of the launches that make the pool's sanitised copies
    return [int(l[2]) for l in log() if l[0] == "pool"]

def on_device(a):
    p = C.c_void_p()
    assert fake.cudaMalloc(C.byref(p), C.c_size_t(a.nbytes)) == OK
    C.memmove(p, a.ctypes.data, a.nbytes)
    return p

def pool(n, each):
    return np.arange(n + 1, dtype=np.uint64) * each, np.full(max(n * each, 1), 65, np.uint8)

def set_pool(n, each, device):
    off, data = pool(n, each)
    if not device:
        return lib.k2j_set_strings(ctx, off.ctypes.data, data.ctypes.data, n)
    fake.fake_pool_total(n * each)
    return lib.k2j_set_strings(ctx, on_device(off), on_device(data), n)
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    from kineto_b200 import build
    build.build()
    so = str(tmp_path_factory.mktemp("fake") / "libfake_cudart.so")
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-I" + include,
                    os.path.join(helpers.ROOT, "tests", "native", "fake_cudart.cpp"), "-o", so], check=True)
    return so


def run(fake, body):
    r = subprocess.run([sys.executable, "-c", PRELUDE + textwrap.dedent(body)], cwd=helpers.ROOT, capture_output=True, text=True,
                       env=dict(os.environ, LD_PRELOAD=fake), timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


def test_a_pool_that_does_not_fit_is_never_written_by_a_retry(fake):
    """The workspaces of a larger pool in device memory are allocated during the segmentation.  Where that fails, every
    later try fails the same way or has the room: no launch is told of room that there is not."""
    run(fake, """
        assert set_pool(10, 10, True) == OK and lib.k2j_segment(ctx, None) == OK
        assert all(100 <= r < 10_000 for r in rooms())
        assert set_pool(10, 1 << 20, True) == OK     # its size is learned by the segmentation
        fake.fake_most(1 << 20)
        for again in range(3):
            assert lib.k2j_segment(ctx, None) == CUDA
            assert all(r < 10_000 for r in rooms()), again
        fake.fake_most(1 << 40)
        assert lib.k2j_segment(ctx, None) == OK
        assert [r >= 10 << 20 for r in rooms()] == [True]
    """)


def test_workspaces_that_could_not_be_had_in_set_strings_are_asked_for_again(fake):
    run(fake, """
        fake.fake_most(1_500_000)
        assert set_pool(10, 100_000, False) == CUDA   # (the copy of the pool fits, its sanitised copies do not)
        assert lib.k2j_segment(ctx, None) == CUDA and rooms() == []
        fake.fake_most(1 << 40)
        assert lib.k2j_segment(ctx, None) == OK
        assert [r >= 1_000_000 for r in rooms()] == [True]
    """)


def test_a_setter_that_fails_leaves_no_arrays_of_its_kind(fake):
    """The staged copies of the call before are gone by then: nothing may read them."""
    run(fake, """
        def ops(n):
            cols = {name: np.zeros(n, np.int64) for name in ("start_ns", "end_ns", "id", "device", "resource", "thread", "type", "name", "flow_id", "flow_info")}
            off = np.zeros(n + 1, np.uint32)
            keep.append((cols, off))
            return lib.k2j_set_ops(ctx, C.byref(api.Ops(n, *[a.ctypes.data for a in cols.values()], off.ctypes.data, None)))

        def cupti(n):
            data, table = np.zeros(n, np.uint8), np.array([0, n], np.uint64)
            return lib.k2j_set_cupti(ctx, data.ctypes.data, n, table.ctypes.data, 1)

        keep, info = [], api.SegmentInfo()
        assert set_pool(10, 10, False) == OK and ops(10) == OK and cupti(4096) == OK
        assert lib.k2j_segment(ctx, C.byref(info)) == OK and info.n_ops == 10
        assert sum("k_seg_chunks" in l[1] for l in log() if l[0] == "launch") == 1
        fake.fake_most(1 << 16)
        assert set_pool(100_000, 1, False) == CUDA and ops(100_000) == CUDA and cupti(1 << 20) == CUDA
        fake.fake_most(1 << 40)
        log()
        assert lib.k2j_segment(ctx, C.byref(info)) == OK and info.n_ops == 0
        assert sum("k_seg_chunks" in l[1] for l in log() if l[0] == "launch") == 0
        assert set_pool(100_000, 1, False) == OK and ops(100_000) == OK and cupti(1 << 20) == OK
        assert lib.k2j_segment(ctx, C.byref(info)) == OK and info.n_ops == 100_000
    """)


def test_arrays_in_device_memory_are_read_behind_the_default_stream(fake):
    """A pool's offsets and the metadata entries in device memory may still be in the making on the legacy default stream:
    either a blocking copy has waited for it, or the context's stream does."""
    run(fake, """
        def ordered():
            lines, recorded = log(), set()
            for l in lines:
                if l[0] == "record" and l[2] == "1":   # cudaStreamLegacy
                    recorded.add(l[1])
            return any(l[0] == "copy_and_wait" or (l[0] == "wait" and l[1] in recorded) for l in lines)

        cols = [on_device(np.zeros(8, np.int64)) for _ in range(10)]
        off, md = on_device(np.arange(9, dtype=np.uint32)), on_device(np.zeros(8 * 4, np.uint64))
        log()
        for trace in range(3):
            assert set_pool(10, 10, True) == OK and ordered(), trace
            assert lib.k2j_set_ops(ctx, C.byref(api.Ops(8, *cols, off, md))) == OK and ordered(), trace
            assert lib.k2j_segment(ctx, None) == OK
            log()
    """)


def test_the_emit_pass_spreads_over_the_sms_that_the_gpu_has(fake):
    """A trace that one wave holds gets the smallest blocks that still make one wave: two an SM of (here) 132."""
    run(fake, """
        def threads(n):
            cols = [np.zeros(n, np.int64) for _ in range(10)]
            off = np.zeros(n + 1, np.uint32)
            assert lib.k2j_set_ops(ctx, C.byref(api.Ops(n, *[a.ctypes.data for a in cols], off.ctypes.data, None))) == OK
            log()
            fake.fake_scan_total(100 * n)
            assert lib.k2j_run(ctx, C.byref(api.Result())) == OK
            (block,) = [int(l[3]) for l in log() if l[0] == "launch" and "k_eventsILb1ELb0E" in l[1]]
            return block

        assert [threads(132 * 2 * k + more) for k, more in ((1, 0), (64, 0), (64, 1), (96, 0), (96, 1), (320, 0), (320, 1))] == [64, 64, 96, 96, 128, 320, 320]
    """)


def test_text_that_leaves_slab_by_slab_takes_no_hand_over(fake):
    """What the size pass works out for the emit pass is kept where the text is kept; the calls that bound memory hold a few
    words an event."""
    run(fake, """
        n = 1 << 20
        columns = np.zeros(13, np.uint64)
        columns[[1, 12]] = n              # kernel records, records that own an event
        fake.fake_columns(C.c_void_p(columns.ctypes.data), 13)
        data, table = np.zeros(4096, np.uint8), np.array([0, 4096], np.uint64)
        assert lib.k2j_set_cupti(ctx, data.ctypes.data, 4096, table.ctypes.data, 1) == OK
        fake.fake_scan_total(1 << 20)
        text, result = np.zeros(1 << 20, np.uint8), api.Result()
        largest = []
        for slabs in (True, False):
            log()
            assert lib.k2j_segment(ctx, None) == OK
            if slabs:
                assert lib.k2j_emit_to_host(ctx, text.ctypes.data, text.nbytes, 0, C.byref(result)) == OK
            else:
                assert lib.k2j_emit(ctx, C.byref(result)) == OK
            lines = log()
            assert sum("k_events" in l[1] for l in lines if l[0] == "launch") >= 1
            largest.append(max([int(l[2]) for l in lines if l[0] == "alloc"], default=0))
        assert largest[0] < 16 * n and largest[1] >= 64 * n
    """)


def test_a_failed_allocation_is_reported_once(fake):
    """The runtime holds the error of a failed call until it is asked for; a later run that has its memory is not refused for it."""
    run(fake, """
        n = 1 << 16
        cols, off = [np.zeros(n, np.int64) for _ in range(10)], np.zeros(n + 1, np.uint32)
        ops = api.Ops(n, *[a.ctypes.data for a in cols], off.ctypes.data, None)
        for most, want in ((1 << 16, CUDA), (1 << 40, OK)):
            fake.fake_most(most)
            assert lib.k2j_set_ops(ctx, C.byref(ops)) == want
        fake.fake_scan_total(100 * n)
        assert lib.k2j_run(ctx, C.byref(api.Result())) == OK
    """)
