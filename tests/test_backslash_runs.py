"""Runs of backslashes over many warps' words, tiles and chunks of a load: the
index equals the sequential definition, and a run costs time in proportion to
its length."""

from __future__ import annotations

import time

import numpy as np
import pytest

import gpjson_b200 as gj
from oracle import oracle

TILE = 16384
OBJ = b'{"a":[1,{"b":"x,]"}],"c":"y"}\n'


def value_of(run: int, before: int) -> bytes:
    """A line whose string value is `run` backslashes (and a quote they escape, where they are odd), `before` bytes
    into the input."""
    pad = b" " * (before - 7)
    return pad + b'\n{"a":"' + b"\\" * run + (b'"' if run & 1 else b"") + b'","b":[{}]}\n' + OBJ


def equal(f, want: oracle.Index, levels: int) -> None:
    assert np.array_equal(f.newline_index(), want.newlines)
    assert np.array_equal(f.string_index(), want.strings)
    assert np.array_equal(f.leveled_bitmaps(levels), want.levels)


@pytest.mark.gpu
@pytest.mark.parametrize("run", [15, 16, 17, 2047, 2048, 2049, 4096, TILE - 16, TILE - 15, TILE - 1, TILE, TILE + 1, 2 * TILE - 16,
                                 2 * TILE, 2 * TILE + 1, 5 * TILE + 64, 40 * TILE + 3])
def test_runs_equal_the_sequential_definition(gpjson, run):
    for before in (7, 8, 2048, TILE - 1, TILE, TILE + 1, TILE + 2049, 3 * TILE - 16):
        data = value_of(run, before)
        want = oracle.Index(data, 4)
        f = gpjson.load_bytes(data)
        try:
            for _ in range(2):
                f.build_index(4)
                equal(f, want, 4)
        finally:
            f.release()


@pytest.mark.gpu
@pytest.mark.parametrize("run", [1, TILE - 1, TILE, TILE + 1, 3 * TILE, 3 * TILE + 1])
def test_runs_from_the_first_byte(gpjson, run):
    for rest in (b'"{\n' + OBJ * 3, b'{"a":1}\n' + OBJ, b""):
        data = b"\\" * run + rest
        want = oracle.Index(data, 4)
        f = gpjson.load_bytes(data)
        try:
            f.build_index(4)
            equal(f, want, 4)
        finally:
            f.release()


@pytest.mark.gpu
def test_runs_in_a_batch(gpjson):
    data = [value_of(run, before) for run, before in ((3 * TILE, 8), (3 * TILE + 1, 9), (TILE, TILE), (40, 2048))]
    want = [oracle.query(d, ["$.b[0]", "$.c"]) for d in data]
    files = [gpjson.load_bytes(d) for d in data]
    b = gpjson.batch()
    try:
        items = [b.add(f, ["$.b[0]", "$.c"]) for f in files]
        b.run()
        for item, w in zip(items, want):
            assert np.array_equal(b.result(item), w)
    finally:
        b.release()
        for f in files:
            f.release()


@pytest.mark.gpu
@pytest.mark.parametrize("run", [33 << 20, (33 << 20) + 1])
def test_long_runs_take_little_time(gpjson, run):
    """Over the border of two chunks of a load too (60 MiB)."""
    data = value_of(run, 40 << 20)
    want = oracle.Index(data, 4)
    queries = [gj.compile_path("$.b[0]")]
    f, got = gpjson.load_bytes_query(data, 4, queries)
    try:
        equal(f, want, 4)
        assert np.array_equal(got, oracle.query(data, ["$.b[0]"]))
        start = time.perf_counter()
        f.build_index(4)
        taken = time.perf_counter() - start
        equal(f, want, 4)
        assert taken < 0.25, taken  # some thousand tiles, a few microseconds each
    finally:
        f.release()
