"""A deeper index that does not fit the device leaves no index behind, and the
file is indexed again when it is next needed.  In a process of its own: other
contexts' pools give unused memory back to one that runs out."""

from __future__ import annotations

import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
PROGRAM = """
import numpy as np
import torch

import gpjson_b200 as gj
from gpjson_b200 import datagen

MIB = 1 << 20


def refused(call) -> bool:
    try:
        call()
    except gj.GPJSONException:
        return True
    return False


dev = torch.from_numpy(datagen.tweets(256 * MIB, seed=datagen.SEED_BASE + 3)).cuda()
torch.cuda.synchronize()
g = gj.GPJSON(0)
f = g.from_device(dev.data_ptr(), dev.numel(), keepalive=dev)
f.build_index(1)
query = [gj.compile_path("$.id")]
want = f.run(query)
hog = torch.empty(torch.cuda.mem_get_info()[0] - 256 * MIB, dtype=torch.uint8, device="cuda")
assert refused(lambda: f.build_index(16)), "512 MiB of bitmaps"
assert refused(lambda: f.run(query)), "no index any more"
assert np.array_equal(f.query_paths(["$.id"]), want)
del hog
torch.cuda.empty_cache()
f.build_index(16)
assert np.array_equal(f.run(query), want)
f.release()
g.close()
print("as before")
"""


@pytest.mark.gpu
def test_levels_that_do_not_fit():
    done = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0 and done.stdout.strip() == "as before", done.stdout + done.stderr
