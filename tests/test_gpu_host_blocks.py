"""Host memory of gathered values that other values hold or have given back,
and files at the edges of the slices they are read in."""

from __future__ import annotations

import numpy as np
import pytest

from gpjson_b200 import datagen


@pytest.mark.gpu
@pytest.mark.parametrize("held", [0, 1, 7])  # 7 of about 13 MiB: some beyond the page-locked 64 MiB
def test_values_held_and_dropped(gpjson, held):
    data = datagen.tweets(24 << 20, seed=datagen.SEED_BASE + 91)
    f = gpjson.load_bytes(data)
    try:
        offsets = f.query_paths(["$.user"])[0].reshape(-1, 2)
        want = b"".join(data[a:b].tobytes() for a, b in offsets if a >= 0)
        assert len(want) > 8 << 20
        kept = [f.query_values(["$.user"]) for _ in range(held)]
        for path in ("$.id", "$.user", "$.text", "$.user"):  # blocks of other sizes in between
            last = f.query_values([path])
        assert last.data == want
        assert all(v.data == want for v in kept)
        lengths = np.diff(last.offsets)
        assert np.array_equal(lengths, np.where(offsets[:, 0] >= 0, offsets[:, 1] - offsets[:, 0], 0))
    finally:
        f.release()


@pytest.mark.gpu
@pytest.mark.parametrize("size", [1, (1 << 20) - 1, 1 << 20, (1 << 20) + 1, (64 << 20) - 1, 64 << 20, (64 << 20) + 1,
                                  (130 << 20) + 12345])
def test_file_slices(gpjson, tmp_path, size):
    """The file's bytes come back as the values of its lines."""
    width = 4096
    lines = np.full((size // width + 1, width), ord("x"), dtype=np.uint8)
    prefix, suffix = b'{"v":"', b'"}\n'
    lines[:, :len(prefix)] = np.frombuffer(prefix, np.uint8)
    lines[:, -len(suffix):] = np.frombuffer(suffix, np.uint8)
    digits = np.char.zfill(np.arange(len(lines)).astype(f"S{9}"), 9)
    lines[:, 8:17] = np.frombuffer(digits.tobytes(), np.uint8).reshape(-1, 9)
    data = lines.reshape(-1)[:size]
    path = tmp_path / "slices.ldjson"
    data.tofile(path)
    f = gpjson.open(path)
    g = gpjson.load_bytes(data)
    try:
        assert f.size == size
        got, want = f.query_values(["$.v"]), g.query_values(["$.v"])
        assert got.data == want.data
        assert np.array_equal(got.offsets, want.offsets) and np.array_equal(got.kinds, want.kinds)
        whole = size // width
        inner = lines[:whole, len(prefix) - 1:-2].tobytes()
        assert got.data[:len(inner)] == inner
    finally:
        f.release()
        g.release()
