"""gpj_tuning.long_line_bytes: a value that is set is the one that counts, the
library's choice stays where it is not."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from gpjson_b200 import _lib
from oracle import oracle

DATA = b"".join(b'{"a":%d,"b":[1,%d]}\n' % (i, i) for i in range(500))


@pytest.mark.gpu
def test_set_values_count(gpjson):
    """Few (line, query) pairs: the library gives each a warp, in one launch; where the line length is set, a launch
    for the short lines is followed by one for the long, and with -1 by none."""
    want = oracle.query(DATA, ["$.a", "$.b[1]"])
    f = gpjson.load_bytes(DATA)
    b = gpjson.batch()
    item = b.add(f, ["$.a", "$.b[1]"])

    def launches() -> tuple[int, int]:
        before = gpjson.kernel_launches()
        assert np.array_equal(f.query_paths(["$.a", "$.b[1]"]), want)
        between = gpjson.kernel_launches()
        b.run()
        assert np.array_equal(b.result(item), want)
        return between - before, gpjson.kernel_launches() - between

    try:
        f.query_paths(["$.a", "$.b[1]"])
        for value, per_query in ((0, 1), (65536, 2), (8192, 2), (262144, 2), (-1, 1), (0, 1), (65536, 2)):
            gpjson.set_tuning(long_line_bytes=value)
            assert gpjson.tuning()["long_line_bytes"] == (value or 65536)
            for _ in range(3):  # (a batch's query phase is replayed from the third run on)
                assert launches() == (per_query, per_query), value
        gpjson.set_tuning(long_line_bytes=0)
        # other values set, this one left: still the library's choice
        gpjson.set_tuning(query_ctas_per_sm=3)
        assert launches() == (1, 1)
        raw = _lib.Tuning()
        lib, h = gpjson._native.lib, gpjson._native.h
        assert lib.gpj_get_tuning(h, ctypes.byref(raw)) == 0
        raw.query_ctas_per_sm = 0
        assert lib.gpj_set_tuning(h, ctypes.byref(raw)) == 0
        assert launches() == (1, 1)
        raw = _lib.Tuning(65536, 0, 0, 0, 0)
        assert lib.gpj_set_tuning(h, ctypes.byref(raw)) == 0
        assert launches() == (2, 2)
        gpjson.set_tuning(query_ctas_per_sm=0)  # a set value stays set
        assert launches() == (2, 2)
    finally:
        gpjson.set_tuning(long_line_bytes=0, query_ctas_per_sm=0)
        b.release()
        f.release()
