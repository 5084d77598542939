"""The standalone index kernel (index_tiles.cu): its word arithmetic on the
host, and its tiles' edges on the GPU against the oracle."""
import ctypes
import random

import numpy as np
import pytest

from oracle import oracle

TILE = 16384


@pytest.mark.parametrize("levels", [4, 8, 16])
def test_bit_parallel_level_split(hostsim, levels):
    """split_half equals the loop over cuts wherever the range check accepts
    the word, and marks the bytes at level -1."""
    fn = hostsim.hs_split_word
    fn.restype = ctypes.c_int
    P = ctypes.c_void_p
    fn.argtypes = [ctypes.c_int, ctypes.c_uint64, ctypes.c_uint64, ctypes.c_uint64, ctypes.c_int, P, P, P]
    halves, loop, minus = (np.zeros(n, dtype=np.uint64) for n in (16, 16, 1))
    r = random.Random(levels)
    accepted = 0
    for trial in range(6000):
        density = r.choice([0.02, 0.1, 0.3, 0.9])
        kinds = [r.choice("[]") if r.random() < density else r.choice(", ") for _ in range(64)]
        if trial % 5 == 0:
            kinds[31], kinds[32] = r.choice("[],"), r.choice("[],")
        masks = [sum(1 << i for i, k in enumerate(kinds) if k in want) for want in ("[", "]", "[],")]
        depth = r.randint(-levels - 1, 2 * levels)
        ok = fn(levels, *masks, depth, halves.ctypes.data, loop.ctypes.data, minus.ctypes.data)
        opens, closes = kinds.count("["), kinds.count("]")
        assert ok == (depth + opens < 2 * levels - 1 and depth - closes >= -levels)
        if not ok:
            continue
        accepted += 1
        assert np.array_equal(halves[:levels], loop[:levels])
        d, at_minus_one = depth, 0
        for i, k in enumerate(kinds):
            d += k == "["
            at_minus_one |= (d == -1) << i
            d -= k == "]"
        assert int(minus[0]) == at_minus_one
    assert accepted > 1000


def test_classification_of_exchanged_halves(hostsim):
    fn = hostsim.hs_classify_swapped
    fn.restype, fn.argtypes = None, [ctypes.c_void_p, ctypes.c_int64, ctypes.c_void_p]
    data = np.random.default_rng(3).permutation(np.repeat(np.arange(256, dtype=np.uint8), 64))
    got, want = (np.zeros(len(data) // 64 * 7, dtype=np.uint64) for _ in range(2))
    fn(data.ctypes.data, len(data) // 64, got.ctypes.data)
    hostsim.hs_classify(data.ctypes.data, len(data) // 64, want.ctypes.data)
    assert np.array_equal(got, want)


def test_escapes_and_prefix_xor(hostsim):
    U, C = ctypes.c_uint64, ctypes.c_uint32
    for name, args, res in (("hs_escaped_bytes", [U, C], U), ("hs_trailing_run_odd", [U], ctypes.c_int),
                            ("hs_prefix_xor", [U, ctypes.c_int], U)):
        getattr(hostsim, name).argtypes, getattr(hostsim, name).restype = args, res
    r = random.Random(5)
    for trial in range(4000):
        bs = r.getrandbits(64) & r.getrandbits(64) if trial % 2 else r.getrandbits(64) | r.getrandbits(64)
        bs = r.choice([bs, bs, 0, ~0 & (1 << 64) - 1, bs | 1, bs | 1 << 63, bs & ~1])
        for cin in (0, 1):
            out = C()
            want = hostsim.hs_escaped_mask(bs, cin, ctypes.byref(out))
            assert hostsim.hs_escaped_bytes(bs, cin) & ~bs == want & ~bs
            if bs != (1 << 64) - 1:
                assert hostsim.hs_trailing_run_odd(bs) == out.value
        assert hostsim.hs_prefix_xor(bs, 1) == hostsim.hs_prefix_xor(bs, 0)


def _edge_inputs():
    """Line ends, long lines, escapes and strings placed around tile edges."""
    obj = b'{"a":[1,{"b":"x,]\\\\"}],"c":"y"}'
    for shift in (-65, -64, -1, 0, 1, 15, 16, 64):  # the line end before, at and after a tile edge
        yield f"line_end{shift}", obj + b" " * (TILE + shift - len(obj)) + b"\n" + obj + b"\n" + obj
    for n in (1, 15, 16, 17, 63, 64, 65, TILE - 1, TILE, TILE + 1, TILE + 16, 2 * TILE + 63):  # sizes
        yield f"size{n}", ((obj + b"\n") * (n // len(obj) + 1))[:n]
    for run in (1, 2, 15, 16, 17, 40, TILE, TILE + 1):  # backslash runs that end at, before and after an edge
        for end in (0, 1, 5):
            head = b'\n{"a":"'
            data = obj + b" " * (2 * TILE + end - run - len(obj) - len(head)) if 2 * TILE > run + 100 else obj
            yield f"run{run}_{end}", data + head + b"\\" * run + b'\\"' * (run & 1) + b'","b":[{}]}\n' + obj
    long = b'{"k":[' + b'{"s":"[\\\"","t":[1,2]},' * 3000 + b"0]}"  # lines over several tiles, nested and in strings
    yield "long_lines", (obj + b"\n") * 40 + long + b"\n" + obj + b"\n" + long + b"\n" + long
    yield "long_string", obj + b'\n{"s":"' + b"{[,:" * 20000 + b'","t":[]}\n' + obj + b"\n"
    yield "deep", (b"[" * 40 + b"1" + b"]" * 40 + b"\n" + obj + b"\n") * 300
    yield "deeper", (b"[" * 5000 + b"1,2" + b"]" * 5000 + b"\n") * 8
    yield "blank", b"\n" * (3 * TILE + 7)
    yield "one_open_line", b'{"a":[' + b"1," * 40000
    # not NDJSON: what the host indexes again with the exact kernel
    yield "pretty", b'{\n  "a": [\n    1,\n    2\n  ]\n}\n' * 4000
    yield "newline_in_string", (obj + b"\n") * 700 + b'{"s":"' + b"ab\n" * 9000 + b'"}\n' + (obj + b"\n") * 700
    yield "unbalanced_at_an_edge", obj + b" " * (TILE - 20 - len(obj)) + b"]" + b" " * 40 + b"\n" + (obj + b"\n") * 900


@pytest.mark.gpu
@pytest.mark.parametrize("levels", [1, 4, 5, 16])
def test_tile_edges(gpjson, levels):
    """String index, leveled bitmaps and newline index equal the sequential
    definition at the edges of tiles, twice over on one file."""
    for name, data in _edge_inputs():
        want = oracle.Index(data, levels)
        f = gpjson.load_bytes(data)
        try:
            for _ in range(2):
                f.build_index(levels)
                assert np.array_equal(f.newline_index(), want.newlines), name
                assert np.array_equal(f.string_index(), want.strings), name
                assert np.array_equal(f.leveled_bitmaps(levels), want.levels), name
        finally:
            f.release()


@pytest.mark.gpu
@pytest.mark.parametrize("levels", [1, 4, 7, 8, 12, 16])
def test_levels_above_the_marked_ones(gpjson, levels):
    """Lines whose nesting wanders around and far above the marked levels."""
    r = random.Random(levels)
    lines = []
    for _ in range(400):
        depth, top, line = 0, r.choice([3, levels, levels + 3, 2 * levels + 9, 200]), []
        for _ in range(r.choice([10, 100, 3000])):
            up = r.random() < (0.7 if depth < top else 0.3)
            line.append(r.choice(["[", "{", ",[", ', "[:]", {']) if up or depth == 0 else r.choice(["]", "}", ",]", " ] "]))
            depth += 1 if up or depth == 0 else -1
            if r.random() < 0.3:
                line.append(r.choice([",", ":", " " * r.randint(1, 90)]))
        lines.append("".join(line) + "]" * depth)
    data = "\n".join(lines).encode()
    want = oracle.Index(data, levels)
    f = gpjson.load_bytes(data)
    try:
        f.build_index(levels)
        assert np.array_equal(f.newline_index(), want.newlines)
        assert np.array_equal(f.string_index(), want.strings)
        assert np.array_equal(f.leveled_bitmaps(levels), want.levels)
    finally:
        f.release()
