"""find_value's thread-per-line and warp-per-line kernels around the rules that
choose between them, and their key searches on every layout of a key, against
the oracle."""
import ctypes
import random

import numpy as np
import pytest

from oracle import oracle

KEYS = ["a", "ab", "abc", "lang", "xlang", "k\\\\\"q", "e\\\\\\\\", "with space"]
PATHS = ["$.a", "$.ab", "$.abc", "$.lang", "$['k\\\"q']", "$['with space']", "$.o.lang", "$.o.a", "$.v[0]", "$.v[7]",
         "$.v[60]", "$.v[1:3]", "$.o.v[2].a", "$.missing"]


def _object(r: random.Random, depth: int, items: int) -> str:
    def value(d):
        if d and r.random() < 0.3:
            return _object(r, d - 1, r.randint(0, 4))
        if d and r.random() < 0.4:
            items = 70 if r.random() < 0.03 else r.choice([0, 1, 3, 8])
            return "[" + r.choice([",", " , "]).join(value(min(d - 1, items < 9)) for _ in range(items)) + "]"
        return r.choice(["1", "null", '"a:b"', '"\\\\"', '"x\\"lang\\":3"', '""', "-2.5e3"])

    keys = [r.choice(KEYS).replace("\\\\", "\\") for _ in range(items)] + r.sample(["o", "v", "lang", "a"], 2)
    r.shuffle(keys)
    gap = lambda: r.choice(["", "", "", " ", "\t "])  # noqa: E731
    return "{" + ",".join(f'{gap()}"{k}"{gap()}:{gap()}{value(depth)}' for k in keys) + "}"


def _lines(lines: int, mean: int, seed: int) -> bytes:
    """`lines` lines of about `mean` bytes (blanks or a long member fill them up), the last without a newline."""
    r = random.Random(seed)
    out = []
    for _ in range(lines):
        line = _object(r, 2, r.randint(0, 6)) if mean > 20 else _object(r, 0, r.randint(0, 2))
        short = mean - len(line)
        if short > 0 and r.random() < 0.5:
            line = '{"pad":' + r.choice(['"' + "x" * short + '"', "[" + "1," * (short // 2) + "0]"]) + "," + line[1:]
        elif short > 0:
            line += " " * short
        out.append(line)
    return "\n".join(out).encode()


def _marks(data: np.ndarray, strings: np.ndarray, r: random.Random) -> tuple[np.ndarray, np.ndarray]:
    """The standalone index kernel's key marks, and its odd words with some more set at random (allowed)."""
    n, words = data.size, strings.size
    state = np.unpackbits(strings.view(np.uint8), bitorder="little")[:n].astype(bool)
    before = np.concatenate([[False], state[:-1]])
    colon = (data == ord(":")) & ~state
    closing = np.concatenate([[False], (before & ~state)[:-1]])
    odd = (data == ord("\\")) | (colon & ~closing)
    bits = np.zeros(words * 64, dtype=np.uint8)
    bits[:n] = colon | (state & ~before)
    marks = np.packbits(bits, bitorder="little").view(np.uint64).copy()
    flags = np.zeros(((words + 31) // 32 * 32, 64), dtype=bool)
    flags.reshape(-1)[:n] = odd
    extra = np.array([r.random() < 0.1 for _ in range(flags.shape[0])])
    return marks, np.packbits(flags.any(axis=1) | extra, bitorder="little").view(np.uint32).copy()


def test_key_search_by_length(hostsim):
    """Judging key candidates by length (marks and odd words), with the
    queries as decoded programs, equals the oracle: keys of every length up to past the limit, with blanks, quotes and
    backslashes in and around them, at every offset to the 64-byte words, in
    well-formed and broken lines."""
    fn = hostsim.hs_find_values_marks
    P, L = ctypes.c_void_p, ctypes.c_int64
    fn.restype, fn.argtypes = None, [P, L, P, L, P, P, P, ctypes.c_int, P, P, P, ctypes.c_int]
    r = random.Random(8)
    names = KEYS + ["z" * n for n in (1, 30, 58, 59, 60, 61, 62, 63, 64, 65, 130)] + ["a\\\\", '\\"lang']
    hits = 0
    for trial in range(150):
        lines = []
        for _ in range(r.randint(1, 8)):
            line = _object(r, 2, r.randint(0, 4))
            for _ in range(r.randint(0, 6)):
                name = r.choice(names).replace("\\\\", "\\")
                member = f'"{name}"{r.choice(["", "", " "])}:{r.choice(["1", "[2,3]", _object(r, 1, 1)])}'
                line = "{" + member + "," + line[1:]
            if r.random() < 0.2:
                k = r.randrange(len(line))
                line = line[:k] + r.choice('{}[]:,"\\ a') + line[k + 1:]
            lines.append(" " * r.randint(0, 3) + line)
        data = np.frombuffer("\n".join(lines).encode(), dtype=np.uint8)
        for path in PATHS + [f"$['{n}']" for n in names[8:-2]] + ["$['a\\\\']", "$['\\\"lang']", "$[',\"a']"]:
            try:
                ir, depth, slots = oracle.compile_path(path)
            except Exception:
                continue
            idx = oracle.Index(data, depth)
            want = oracle.find_value(data, idx.newlines, idx.strings, idx.levels, depth, ir, slots)
            hits += int((want >= 0).sum())
            marks, odd = _marks(data, idx.strings, r)
            code = np.frombuffer(ir, dtype=np.uint8)
            for how in (0, 1, 2):
                got = np.full_like(want, 7)
                fn(data.ctypes.data, data.size, idx.newlines.ctypes.data, len(idx.newlines), idx.strings.ctypes.data,
                   idx.levels.ctypes.data, code.ctypes.data, slots, got.ctypes.data, marks.ctypes.data,
                   odd.ctypes.data, how)
                assert np.array_equal(got, want), (path, how, data.tobytes())
    assert hits > 2000


@pytest.mark.gpu
@pytest.mark.parametrize("lines,mean", [(1, 40), (33, 100), (580, 90), (590, 90), (1170, 60), (1500, 20), (70, 4000), (70, 4300),
                                        (40, 9000), (5, 70000), (3, 400000)])
def test_thread_and_warp_kernels(gpjson, lines, mean):
    """The number of (line, query) pairs (8192) and the mean line length (4096
    bytes) choose the kernel, 8 KiB the lines handed over; every choice, forced
    or not, equals the oracle, singly and in a batch."""
    data = _lines(lines, mean, seed=lines + mean)
    want = oracle.query(data, PATHS)
    f = gpjson.load_bytes(data)
    try:
        for long_line_bytes in (65536, 64, -1):
            gpjson.set_tuning(long_line_bytes=long_line_bytes)
            try:
                assert np.array_equal(f.query_paths(PATHS), want), long_line_bytes
                b = gpjson.batch()
                try:
                    item = b.add(f, PATHS)
                    b.run()
                    assert np.array_equal(b.result(item), want), long_line_bytes
                finally:
                    b.release()
            finally:
                gpjson.set_tuning(long_line_bytes=0)
    finally:
        f.release()
