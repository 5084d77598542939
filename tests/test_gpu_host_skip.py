"""Loads that evaluate queries while later bytes are still on their way: a
query whose whitespace skip runs from a blank line into bytes that have not
arrived is evaluated again, and never reads what the memory held before."""

from __future__ import annotations

import numpy as np
import pytest

import gpjson_b200 as gj
from oracle import oracle

CHUNK = 2048 * 30720  # bytes a load copies at a time
PATHS = ["$[0]", "$[1]", "$.a"]


@pytest.mark.gpu
@pytest.mark.parametrize("blanks", [1000, CHUNK, 2 * CHUNK - 8, 2 * CHUNK - 7, 2 * CHUNK - 6, 3 * CHUNK + 5])
def test_skip_past_the_loaded_bytes(gpjson, blanks):
    data = np.frombuffer(b"[1,2]\n\n" + b" " * blanks + b"[7]\n[8,[9]]\n" + b'{"a":3}\n' * 9, dtype=np.uint8)
    data = np.concatenate([data, np.full(max(0, 2 * CHUNK + 99 - data.size), ord(" "), dtype=np.uint8)])
    want = oracle.query(data, PATHS)
    assert want[0, 1, 0, 0] == 7 + blanks + 1  # the blank line's answer lies after the blanks
    queries = [gj.compile_path(p) for p in PATHS]
    # what the pool's memory holds when the load takes it
    gpjson.load_bytes(np.full(data.size, ord("["), dtype=np.uint8)).release()
    f, got = gpjson.load_bytes_query(data, 2, queries)
    try:
        assert np.array_equal(got, want)
        assert np.array_equal(f.run(queries), want)
    finally:
        f.release()
