"""Batches whose results are copied to the host in several groups of files,
run as launches, captured and replayed."""

from __future__ import annotations

import numpy as np
import pytest

from gpjson_b200 import datagen

PATHS = ["$.k", "$.a[1]", "$.a[0:3]", "$.none"]


def short_lines(count: int, first: int) -> bytes:
    return b"".join(b'{"k":%d,"a":[%d,"x"]}\n' % (i, i % 7) for i in range(first, first + count))


@pytest.mark.gpu
@pytest.mark.parametrize("files", [1, 3, 9])
def test_groups(gpjson, files):
    # a file's 60,000 lines, 4 paths of up to 3 slots: 11.5 MB of results
    data = [short_lines(60_000 - 7 * i, 100 * i) for i in range(files)]
    data.insert(1, datagen.adversarial(3 << 20, seed=datagen.SEED_BASE + 31).tobytes())  # a warp per line
    data.insert(1, b"")
    data.append(short_lines(3, 5))
    data.append(b'{"k":"' + b"y" * 90_000 + b'"}\n{"k": 3}')
    loaded = [gpjson.load_bytes(d) for d in data]
    want = [f.query_paths(PATHS) for f in loaded]
    b = gpjson.batch()
    try:
        items = [b.add(f, PATHS) for f in loaded]
        for _ in range(4):
            b.run()
            got = [b.result(it) for it in items]
            assert all(np.array_equal(g, w) for g, w in zip(got, want))
            del got
        held = [b.result(it) for it in items]
        b.run()
        assert all(np.array_equal(g, w) for g, w in zip(held, want))
    finally:
        b.release()
        for f in loaded:
            f.release()
