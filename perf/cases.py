"""What the library's speed is measured on: the calls a user's program makes,
over the range of input sizes, line shapes, path sets and options they meet.

``listed()`` names the cases, ``draw(rng)`` gives further ones of the same
ranges; ``prepare`` makes the inputs and the objects such a program keeps,
``run`` makes one pass through the public entry points and returns its
outputs, ``work`` counts the bytes a pass cannot do without.

Every output is a whole number (byte offsets, bitmaps, line counts, value
bytes), so there is nothing to compare against in floating point.

Calls (``call`` of a case):
  index_query  File.index_and_query_device: index and queries of an input
               resident in device memory, results left on the device
  index        gpj_build_index_device: the structural index alone, into the
               caller's device buffers
  query        gpj_query_device: queries on a resident index, results left on
               the device
  request      one request on bytes already on the device: wrap, query_paths,
               results on the host, release
  values       File.query_values on a resident index: matched values gathered
  batch        Batch: many files of uneven size and their queries together
  host         GPJSON.load_bytes_query: page-locked host bytes in, host
               results out, copy, index and queries pipelined
  file         GPJSON.query: a file name and a path in, host results out

Inputs (``data``): the generator's tweet-like lines (about 1.6 KB), its
adversarial lines (100 B-1 MiB, nesting 1-16, backslash runs), and short
records of about 100 bytes (logs, metrics, rows of a table).
"""

from __future__ import annotations

import ctypes
import os
import random
import shutil
import tempfile

import numpy as np
import torch

import gpjson_b200 as gj
from gpjson_b200 import datagen
from gpjson_b200.serve import PATH_POOL

KIB, MIB, GIB = 1 << 10, 1 << 20, 1 << 30

# mean bytes per line of each input, for work()
LINE_BYTES = {"tweets": 1642, "adversarial": 120_000, "records": 117}

TWEET_PATHS = PATH_POOL[:16]
ADVERSARIAL_PATHS = ["$.id"] + PATH_POOL[16:]
RECORD_PATHS = ["$.id", "$.user.lang", "$.user.id", "$.tags[0]", "$.tags[1]", "$.ok", "$.value"]
PATHS = {"tweets": TWEET_PATHS, "adversarial": ADVERSARIAL_PATHS, "records": RECORD_PATHS}

LANGS = ["en", "nl", "de", "fr"]

FOUR = "$.user.lang;$.id;$.user.followers_count;$.entities.hashtags[0].text"


def listed() -> list[dict]:
    return [
        # the benchmark's headline: one 2 GiB file, one index build, four queries
        {"name": "index_query_tweets_2g", "call": "index_query", "data": "tweets", "bytes": 2 * GIB, "levels": 4,
         "paths": FOUR},
        # lines of up to a megabyte, deep nesting, escapes: the benchmark's adversarial file, scaled
        {"name": "index_query_adversarial_1g", "call": "index_query", "data": "adversarial", "bytes": GIB, "levels": 5,
         "paths": "$.a.b.c.d;$.arr[5];$.x[0].y[2].z"},
        # rows of a table or a log: short lines, more lines than any size estimate expects
        {"name": "index_query_records_256m", "call": "index_query", "data": "records", "bytes": 256 * MIB + 77,
         "levels": 2, "paths": "$.user.lang;$.tags[1]"},
        # an extraction job: every path of the 32-path pool over one file, several result slots a line
        {"name": "index_query_32_paths_64m", "call": "index_query", "data": "tweets", "bytes": 64 * MIB, "levels": 6,
         "paths": ";".join(PATH_POOL)},
        # the index alone, at the deepest level count
        {"name": "index_16_levels_256m", "call": "index", "data": "adversarial", "bytes": 256 * MIB - 31, "levels": 16,
         "paths": ""},
        # queries on an index that is already resident
        {"name": "query_resident_512m", "call": "query", "data": "tweets", "bytes": 512 * MIB, "levels": 4,
         "paths": FOUR},
        # single requests, where launches, waits and the host's work count
        {"name": "request_16k", "call": "request", "data": "tweets", "bytes": 16 * KIB + 5, "levels": 2,
         "paths": "$.user.lang"},
        {"name": "request_1m", "call": "request", "data": "tweets", "bytes": 1_000_003, "levels": 4,
         "paths": "$.id;$.text;$.entities.hashtags[0].text"},
        # the matched values themselves, strings of some ten to some hundred bytes
        {"name": "values_128m", "call": "values", "data": "tweets", "bytes": 128 * MIB, "levels": 2,
         "paths": "$.text;$.user.name"},
        # many files of 4 KiB-64 MiB in one batch, three in four tweet-like
        {"name": "batch_48_files", "call": "batch", "data": "mixed", "files": 48, "median": 6_000_000, "levels": 6,
         "paths": ""},
        # input in host memory: the copy over PCIe bounds it
        {"name": "host_query_256m", "call": "host", "data": "tweets", "bytes": 256 * MIB, "levels": 4, "paths": FOUR},
        # the reference's own call: a file name and a path
        {"name": "query_file_64m", "call": "file", "data": "tweets", "bytes": 64 * MIB, "levels": 2,
         "paths": "$.user.lang"},
    ]


def draw(rng: random.Random) -> dict:
    def size(lo: int, hi: int) -> int:
        return int(lo * (hi / lo) ** rng.random()) | 1

    call = rng.choice(["index_query", "index_query", "index", "query", "request", "request", "values", "batch", "host",
                       "file"])
    if call == "batch":
        return {"call": "batch", "data": "mixed", "files": rng.randint(4, 48), "median": size(100_000, 6_000_000),
                "levels": 6, "paths": ""}
    data = rng.choice(["tweets", "tweets", "adversarial", "records"])
    lo, hi = {"index_query": (MIB, GIB), "index": (MIB, 256 * MIB), "query": (MIB, 512 * MIB),
              "request": (4 * KIB, 64 * MIB), "values": (MIB, 128 * MIB), "host": (MIB, 256 * MIB),
              "file": (64 * KIB, 64 * MIB)}[call]
    if data == "records":
        hi = max(lo, hi // 4)  # the results of short lines are as large as the input
    pool = PATHS[data]
    paths = rng.sample(pool, rng.randint(1, min(6, len(pool))))
    depth = max(gj.compile_path(p).max_depth for p in paths)
    levels = rng.choice([depth, max(depth, 4), 8, 16]) if call in ("index_query", "index", "query") else depth
    return {"call": call, "data": data, "bytes": size(lo, hi), "levels": levels, "paths": ";".join(paths)}


# ---- inputs --------------------------------------------------------------------


# Whole lines of each kind, made once; inputs are made of them.
_POOL_BYTES = {"tweets": 16 * MIB, "adversarial": 48 * MIB}
_pools: dict[str, list[bytes]] = {}


def _record_lines() -> list[bytes]:
    r = random.Random(12)
    lines = []
    for _ in range(40_000):
        tags = ",".join(f'"t{r.randrange(1000)}"' for _ in range(r.randint(0, 3)))
        msg = "".join(r.choices(["ab", " ", "c", "\\n", "\\\"", "\\u00e9", "def"], k=r.randint(0, 12)))
        lines.append(f'{{"id":{r.randrange(10**9)},"user":{{"id":{r.randrange(10**6)},"lang":"{r.choice(LANGS)}"}},'
                     f'"tags":[{tags}],"ok":{r.choice(["true", "false"])},"value":{r.random():.4f},"msg":"{msg}"}}\n')
    return [line.encode() for line in lines]


def _lines(data: str) -> list[bytes]:
    if data not in _pools:
        if data == "records":
            _pools[data] = _record_lines()
        else:
            make = datagen.tweets if data == "tweets" else datagen.adversarial
            _pools[data] = make(_POOL_BYTES[data], seed=datagen.SEED_BASE + 1).tobytes().splitlines(keepends=True)
    return _pools[data]


def _input(data: str, nbytes: int, seed: int) -> np.ndarray:
    """Whole lines that fill nbytes, in the seed's order: which lines follows from the size alone, so inputs of one
    size have the same number of lines and values.  What no line fills is blanks, some of them before the first."""
    lines = _lines(data)
    total, shortest = sum(map(len, lines)), min(map(len, lines))
    order = np.random.default_rng(seed)
    repeats, room = divmod(nbytes, total)  # every line, over and over, then as many as still fit
    some = []
    for k in np.random.default_rng(nbytes).permutation(len(lines)):
        if room < shortest:
            break
        if len(lines[k]) <= room:
            some.append(lines[k])
            room -= len(lines[k])
    before = int(order.integers(0, min(room, 256) + 1))
    every = np.frombuffer(b"".join([lines[k] for k in order.permutation(len(lines))]), dtype=np.uint8)
    rest = np.frombuffer(b"".join([some[k] for k in order.permutation(len(some))]), dtype=np.uint8)
    out = np.full(nbytes, 32, dtype=np.uint8)
    out[before:before + repeats * total].reshape(repeats, total)[:] = every
    out[before + repeats * total:][:len(rest)] = rest
    return out


_library = None


def _gpjson() -> "gj.GPJSON":
    """The library object: a program makes one and keeps it."""
    global _library
    if _library is None:
        _library = gj.GPJSON(0)
    return _library


class _Compiled:
    """Compiled paths and the argument arrays of the C entry points."""

    def __init__(self, paths: list[str]):
        self.queries = [gj.compile_path(p) for p in paths]
        self.slots = max(q.num_results for q in self.queries)
        n = len(self.queries)
        self._buffers = [ctypes.create_string_buffer(q.bytecode, len(q.bytecode)) for q in self.queries]
        self.ptrs = (ctypes.c_void_p * n)(*[ctypes.addressof(b) for b in self._buffers])
        self.lens = (ctypes.c_size_t * n)(*[len(q.bytecode) for q in self.queries])


class _TempFile:
    """A file that goes when its state does."""

    def __init__(self, data: np.ndarray):
        self.folder = tempfile.mkdtemp(prefix="gpjson_case_")
        self.name = os.path.join(self.folder, "input.ndjson")
        data.tofile(self.name)

    def __del__(self):
        shutil.rmtree(self.folder, ignore_errors=True)


def prepare(case: dict, seed: int) -> dict:
    g = _gpjson()
    call = case["call"]
    state = {"call": call, "g": g, "paths": [p for p in case["paths"].split(";") if p], "levels": case["levels"]}
    if call == "batch":
        rng = np.random.default_rng(case["files"])
        sizes = np.clip(case["median"] * rng.lognormal(0.0, 1.4, case["files"]), 4 * KIB, 64 * MIB).astype(np.int64)
        state["inputs"], state["requests"] = [], []
        for i, n in enumerate(sizes):
            data = "tweets" if i % 4 else "adversarial"
            host = _input(data, int(n), seed * 64 + i)
            state["inputs"].append(torch.from_numpy(host).cuda())
            picked = rng.choice(len(PATH_POOL), size=int(rng.integers(1, 9)), replace=False)
            state["requests"].append([PATH_POOL[k] for k in picked])
        state["batch"] = g.batch()
        return state
    n = case["bytes"]
    if call == "host":
        pinned = torch.empty(n, dtype=torch.uint8, pin_memory=True)
        pinned.numpy()[:] = _input(case["data"], n, seed)
        state["host"] = pinned.numpy()
        lines = int(np.count_nonzero(state["host"] == 10)) + 1
        state["pinned"] = pinned
        state["compiled"] = _Compiled(state["paths"])
        state["out"] = torch.empty(len(state["paths"]) * lines * state["compiled"].slots * 2, dtype=torch.int64,
                                   pin_memory=True).numpy()
        return state
    host = _input(case["data"], n, seed)
    if call == "file":
        state["file"] = _TempFile(host)
        return state
    state["input"] = dev = torch.from_numpy(host).cuda()
    if call == "request":
        return state
    lines = int(torch.count_nonzero(dev == 10)) + 1
    if call == "index":
        words = (n + 63) // 64
        state["string"] = torch.empty(words, dtype=torch.int64, device="cuda")
        state["leveled"] = torch.empty((case["levels"], words), dtype=torch.int64, device="cuda")
        state["newlines"] = torch.empty(lines, dtype=torch.int64, device="cuda")
        return state
    state["file"] = f = g.from_device(dev.data_ptr(), n, keepalive=dev)
    if call in ("query", "values"):
        f.build_index(case["levels"])
    if call in ("index_query", "query"):
        state["compiled"] = c = _Compiled(state["paths"])
        state["lines"] = lines
        state["out"] = torch.empty((len(c.queries), lines, c.slots, 2), dtype=torch.int64, device="cuda")
    return state


# ---- one pass ------------------------------------------------------------------


def run(state: dict):
    g, call = state["g"], state["call"]
    if call == "index_query":
        c = state["compiled"]
        state["file"].index_and_query_device(c.queries, state["levels"], state["out"].data_ptr(), state["lines"],
                                             c.slots)
        return state["out"]
    if call == "index":
        dev, nl = state["input"], state["newlines"]
        lines = ctypes.c_int64()
        g._native.check(g._native.lib.gpj_build_index_device(
            g._native.h, dev.data_ptr(), dev.numel(), state["levels"], state["string"].data_ptr(),
            state["leveled"].data_ptr(), nl.data_ptr(), nl.numel(), ctypes.byref(lines)))
        return {"string": state["string"], "leveled": state["leveled"], "newlines": nl, "lines": lines.value}
    if call == "query":
        c, out = state["compiled"], state["out"]
        g._native.check(g._native.lib.gpj_query_device(g._native.h, state["file"]._h, len(c.queries), c.ptrs, c.lens,
                                                       c.slots, out.data_ptr(), out.numel()))
        return out
    if call == "request":
        dev = state["input"]
        f = g.from_device(dev.data_ptr(), dev.numel(), keepalive=dev)
        offsets = f.query_paths(state["paths"])
        f.release()
        return offsets
    if call == "values":
        v = state["file"].query_values(state["paths"])
        return {"kinds": v.kinds, "offsets": v.offsets, "data": np.frombuffer(v.data, dtype=np.uint8)}
    if call == "batch":
        batch = state["batch"]
        files = [g.from_device(t.data_ptr(), t.numel(), keepalive=t) for t in state["inputs"]]
        batch.clear()
        for f, paths in zip(files, state["requests"]):
            batch.add(f, paths)
        batch.run()
        results = [batch.result(i) for i in range(len(files))]
        batch.clear()
        for f in files:
            f.release()
        return results
    if call == "host":
        c = state["compiled"]
        f, offsets = g.load_bytes_query(state["host"], state["levels"], c.queries, c.slots, out=state["out"])
        f.release()
        return offsets
    return g.query(state["file"].name, state["paths"]).offsets


def work(case: dict) -> dict:
    """Bytes of one pass: the input read once, the index it leaves and the results written once (for queries on
    a resident index: the newline index and the bitmaps of the levels read once, the results written once)."""
    if case["call"] == "batch":
        # mean of the clipped sizes, about 1.9 medians; four paths of one slot on average
        n = int(case["files"] * 1.9 * case["median"])
        lines = n // LINE_BYTES["tweets"]
        return {"bytes": n + n // 64 * 8 * (1 + case["levels"]) + 8 * lines + 16 * 4 * lines, "flops": 0}
    n, levels = case["bytes"], case["levels"]
    words, lines = (n + 63) // 64, n // LINE_BYTES[case["data"]] + 1
    paths = [p for p in case["paths"].split(";") if p]
    slots = max((gj.compile_path(p).num_results for p in paths), default=0)
    index = words * 8 * (1 + levels) + 8 * lines
    results = 16 * len(paths) * slots * lines
    if case["call"] == "query":
        return {"bytes": index + results, "flops": 0}
    if case["call"] == "values":
        return {"bytes": index + (1 + 8 + 2 * 40) * len(paths) * slots * lines, "flops": 0}
    return {"bytes": n + index + results, "flops": 0}
