"""Parts of the emit pass that compile for the host."""
import ctypes
import os
import re
import subprocess

import numpy as np
import pytest

import helpers


@pytest.fixture(scope="module")
def ec(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("ec") / "libec.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-I" + os.path.join(helpers.ROOT, "kineto_b200", "csrc"),
                    os.path.join(helpers.ROOT, "tests", "native", "emit_check.cpp"), "-o", so], check=True)
    lib = ctypes.CDLL(so)
    lib.ec_long_words.restype = ctypes.c_int64
    lib.ec_long_words.argtypes = [ctypes.c_uint64, ctypes.c_int, ctypes.c_int]
    lib.ec_packed_doubles.restype = ctypes.c_int64
    return lib


@pytest.mark.parametrize("max_len", [0, 7, 8, 15, 40, 100, 700])
def test_long_strings_past_the_window(ec, max_len):
    """Every length and alignment, neighbours written in any order: the plain concatenation of the events."""
    for seed in range(1, 41):
        assert ec.ec_long_words(seed, 150, max_len) == 0, seed


def test_packed_doubles_print_as_the_doubles(ec):
    rng = np.random.default_rng(5)
    v = np.concatenate([rng.random(20000) * 10.0 ** rng.integers(-60, 90, 20000), rng.integers(0, 1 << 53, 20000).astype(np.float64),
                        (rng.random(20000) * 70000).astype(np.float32).astype(np.float64), [1e-46, 9.9e80, 1e81, 0.1, 5e-324, 1e22, 1.0]])
    left = ctypes.c_int64()
    assert ec.ec_packed_doubles(v.ctypes.data_as(ctypes.c_void_p), ctypes.c_int64(len(v)), ctypes.byref(left)) == 0
    assert left.value == int(np.sum((v < 1e-46) | (v >= 1e81)))
    special = np.array([0.0, -0.0, -1.5, np.inf, -np.inf, np.nan])
    assert ec.ec_packed_doubles(special.ctypes.data_as(ctypes.c_void_p), ctypes.c_int64(6), ctypes.byref(left)) == 0
    assert left.value == 6


def test_code_out_of_line_uses_the_sink_without_wide_stores():
    """256-bit stores are right only in a kernel's own code: WindowSink has none, and no function that is called names the other."""
    csrc = os.path.join(helpers.ROOT, "kineto_b200", "csrc")
    src = '#include <string>\n#include "k2j_sink.cuh"\nstatic_assert(!k2j::WindowSink::kWide && k2j::InlineSink::kWide, "");\n'
    r = subprocess.run(["g++", "-std=c++17", "-I" + csrc, "-fsyntax-only", "-x", "c++", "-"], input=src, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    with open(os.path.join(csrc, "k2j_kernels.cuh")) as f:
        text = f.read()
    called = [text[at:text.index("\n}\n", at)] for at in (m.start() for m in re.finditer("__noinline__", text))]
    assert sum("WindowSink" in body for body in called) >= 8
    assert not [body for body in called if re.search(r"InlineSink|Sink<true>|flush<true>|long_words<true>|\bstore32\b", body)]
