"""A resident corpus holds no more device memory than the server counts for it
(no GPU)."""

from __future__ import annotations

import ctypes
import random
import subprocess
from pathlib import Path

import pytest

from gpjson_b200 import serve

SOURCE = '''
#include "index_layout.h"
extern "C" int64_t words(int64_t n, int levels) { return gpj::index_words(n, levels); }
extern "C" int64_t lines(int64_t n, int levels) { return gpj::first_lines(n, levels); }
'''


@pytest.fixture(scope="module")
def layout(tmp_path_factory):
    so = tmp_path_factory.mktemp("layout") / "layout.so"
    csrc = Path(serve.__file__).parent / "csrc"
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", f"-I{csrc}", "-x", "c++", "-o", str(so), "-"],
                   input=SOURCE.encode(), check=True)
    lib = ctypes.CDLL(str(so))
    for fn in (lib.words, lib.lines):
        fn.restype, fn.argtypes = ctypes.c_int64, [ctypes.c_int64, ctypes.c_int]
    return lib


def test_index_within_the_counted_bytes(layout):
    r = random.Random(1)
    sizes = [0, 1, 63, 64, 65, 1023, 1024, 1025, 4095, 4096, 4097, 1 << 20, (1 << 20) + 1, 1 << 31, (1 << 36) + 1]
    sizes += [int(2 ** (r.random() * 40)) for _ in range(2000)]
    for n in sizes:
        for levels in (1, 2, 6, 16):
            assert n + 8 * layout.words(n, levels) <= serve.resident_bytes(n, levels), (n, levels)
            # room for the lines of an input of 300 bytes a line, and some
            assert layout.lines(n, levels) >= min(n + 1, n // 300 + 700)
