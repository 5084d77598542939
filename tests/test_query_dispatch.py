"""find_value's thread-per-line and warp-per-line kernels around the rules that
choose between them, and their key searches on every layout of a key, against
the oracle."""
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
        line = _object(r, 2, r.randint(0, 6))
        short = mean - len(line)
        if short > 0 and r.random() < 0.5:
            line = '{"pad":' + r.choice(['"' + "x" * short + '"', "[" + "1," * (short // 2) + "0]"]) + "," + line[1:]
        elif short > 0:
            line += " " * short
        out.append(line)
    return "\n".join(out).encode()


@pytest.mark.gpu
@pytest.mark.parametrize("lines,mean", [(1, 40), (33, 100), (580, 90), (590, 90), (1170, 60), (70, 4000), (70, 4300),
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
