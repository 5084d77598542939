"""Loads in a context whose memory pool holds no more than they need, with a
file resident beside them: its memory is used again as it is, not mapped
anew."""

from __future__ import annotations

import ctypes
import statistics
import time

import numpy as np
import pytest

import gpjson_b200 as gj
from gpjson_b200 import datagen

PATHS = ["$.user.lang", "$.id", "$.user.followers_count", "$.entities.hashtags[0].text"]
SIZE = 1 << 30


@pytest.mark.gpu
def test_loads_beside_a_resident_file():
    import torch

    pinned = torch.empty(SIZE, dtype=torch.uint8, pin_memory=True)
    data = pinned.numpy()
    datagen.tweets(SIZE, seed=datagen.SEED_BASE + 1, out=data)
    dev = pinned.cuda()
    torch.cuda.synchronize()
    queries = [gj.compile_path(p) for p in PATHS]
    bufs = [ctypes.create_string_buffer(q.bytecode, len(q.bytecode)) for q in queries]
    ptrs = (ctypes.c_void_p * len(queries))(*[ctypes.addressof(b) for b in bufs])
    lens = (ctypes.c_size_t * len(queries))(*[len(q.bytecode) for q in queries])
    g = gj.GPJSON(0)
    try:
        lib, h = g._native.lib, g._native.h
        resident = g.from_device(dev.data_ptr(), SIZE, keepalive=dev)
        for _ in range(2):
            resident.build_index(4)
        out = torch.empty(len(queries) * resident.num_lines * 2, dtype=torch.int64, pin_memory=True).numpy()

        def query(f) -> float:
            start = time.perf_counter()
            g._native.check(lib.gpj_query(h, f._h, len(queries), ptrs, lens, 1, out.ctypes.data, out.size))
            return time.perf_counter() - start

        query(resident)
        want = out.copy()

        # the resident file's results have their memory; a loaded file's are the last that a load takes
        kept = statistics.median(query(resident) for _ in range(8))
        taken = []
        for _ in range(8):
            f, _ = g.load_bytes_query(data, 4, queries, out=out)
            f.release()
            f = g.load_bytes_indexed(data, 4)
            taken.append(query(f))
            assert np.array_equal(out, want)
            f.release()
        loaded = statistics.median(taken[1:])
        assert loaded < 1.15 * kept, (loaded, kept)
        resident.release()
    finally:
        g.close()
