"""Which values get page-locked host memory (no GPU)."""

from __future__ import annotations

import ctypes
import random
import subprocess
from pathlib import Path

import pytest

MIB = 1 << 20
MOST = 64 * MIB


class Store:
    def __init__(self, lib):
        self.lib, self.held = lib, []

    def take(self, size: int) -> tuple[int, int, bool]:
        cap, pinned = ctypes.c_uint64(), ctypes.c_int()
        p = self.lib.vb_take(size, ctypes.byref(cap), ctypes.byref(pinned))
        assert p and cap.value >= size
        ctypes.memset(p, 0x5A, size)
        assert self.lib.vb_locked_bytes() <= MOST
        return p, cap.value, bool(pinned.value)

    def give(self, block) -> None:
        self.lib.vb_give(block[0], block[1], int(block[2]))


@pytest.fixture
def store(tmp_path):
    src = Path(__file__).parent / "hostsim" / "value_blocks.cpp"
    so = tmp_path / "libvalue_blocks.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-o", str(so), str(src)], check=True)
    lib = ctypes.CDLL(str(so))
    U = ctypes.c_uint64
    lib.vb_take.restype, lib.vb_take.argtypes = ctypes.c_void_p, [U, ctypes.POINTER(U), ctypes.POINTER(ctypes.c_int)]
    lib.vb_give.restype, lib.vb_give.argtypes = None, [ctypes.c_void_p, U, ctypes.c_int]
    lib.vb_locks.restype = lib.vb_locked_bytes.restype = ctypes.c_int64
    lib.vb_context(1)
    yield Store(lib)
    lib.vb_context(0)
    assert lib.vb_locked_bytes() == 0


def test_small_values_do_not_hold_the_block_of_large_ones(store):
    store.give(store.take(60 * MIB))
    small = store.take(5000)
    assert small[2] and small[1] <= 2 * MIB
    locks = store.lib.vb_locks()
    large = store.take(60 * MIB)
    assert large[2] and store.lib.vb_locks() == locks  # the same block again
    store.give(large)
    store.give(small)


def test_a_size_that_fits_exactly_is_page_locked(store):
    store.give(store.take(10 * MIB))
    large = store.take(60 * MIB)  # with a quarter to spare it would not fit
    assert large[2]
    store.give(large)


def test_two_sizes_in_turn_are_not_locked_again(store):
    for sizes in ((50, 20), (40, 10), (63, 1), (30, 35)):
        for size in sizes * 2:
            store.give(store.take(size * MIB))
        locks = store.lib.vb_locks()
        for size in sizes * 5:
            block = store.take(size * MIB)
            assert block[2]
            store.give(block)
        assert store.lib.vb_locks() == locks, sizes


def test_random_sizes_held_and_given_back(store):
    r = random.Random(3)
    held = []
    for _ in range(3000):
        if held and r.random() < 0.5:
            store.give(held.pop(r.randrange(len(held))))
        else:
            held.append(store.take(int(2 ** (r.random() * 24))))
    for block in held:
        store.give(block)
