"""A deeper index that does not fit the device leaves no index behind, and the
file is indexed again when it is next needed."""

from __future__ import annotations

import numpy as np
import pytest

import gpjson_b200 as gj
from gpjson_b200 import datagen

SIZE = 256 << 20


@pytest.mark.gpu
def test_levels_that_do_not_fit():
    import torch

    dev = torch.from_numpy(datagen.tweets(SIZE, seed=datagen.SEED_BASE + 3)).cuda()
    torch.cuda.synchronize()
    g = gj.GPJSON(0)
    f = g.from_device(dev.data_ptr(), SIZE, keepalive=dev)
    hog = None
    try:
        f.build_index(1)
        query = [gj.compile_path("$.id")]
        want = f.run(query)
        free = torch.cuda.mem_get_info()[0]
        hog = torch.empty(free - (256 << 20), dtype=torch.uint8, device="cuda")
        with pytest.raises(gj.GPJSONException):
            f.build_index(16)  # 512 MiB of bitmaps
        with pytest.raises(gj.GPJSONException):
            f.run(query)
        assert np.array_equal(f.query_paths(["$.id"]), want)
        del hog
        hog = None
        torch.cuda.empty_cache()
        f.build_index(16)
        assert np.array_equal(f.run(query), want)
    finally:
        del hog
        torch.cuda.empty_cache()
        f.release()
        g.close()
