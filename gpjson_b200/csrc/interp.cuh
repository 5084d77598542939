// Per-line JSONPath bytecode interpreter over the leveled bitmaps.
//
// Semantics follow the reference interpreter find_value
// (gpjson/src/main/resources/com/koenv/gpjson/kernels/find_value.cu:21-263),
// which equals Sequential.findValue (sequential/Sequential.java:130-344).
// Instead of visiting every byte, the scan jumps from one structural bit of
// the current level to the next: bytes without such a bit cannot change the
// interpreter's state while it is searching (find_value.cu skips whole zero
// words for the same reason, :218-222).
//
// Where the reference reads out of bounds or trips a device assert, the
// behaviour below is fixed (marked [bounded]) and the test oracle implements
// the same choice.  __host__ __device__ so the test suite can run it on the
// CPU against the oracle.
#pragma once

#include <cstddef>
#include <cstdint>

#include "word_ops.cuh"

namespace gpj {

// One more than the deepest level a query may reach (16 key/index steps).
constexpr int kLevelSlots = 17;

struct LineView {
    const uint8_t* file;
    int64_t n;
    const uint64_t* string_index;
    const uint64_t* levels;  // [level][level_size], level_size a multiple of 4
    int64_t level_size;
    // Bytes at positions >= hi are not readable through this view (hi = n
    // for the whole file in device memory; a shared-memory view ends at the
    // last byte it holds).  A whitespace skip that reaches hi < n cannot be
    // finished here and the line is reported as deferred.
    int64_t hi;
    // Optional ':' outside strings, indexed like string_index.  When given,
    // a key search jumps only between structural colons and an index search
    // only between the other structural characters.
    const uint64_t* colon;
    // Optional, one bit per word of 64 bytes (32 to an entry, numbered from
    // the file's first byte): then `colon` also has the quotes that open a
    // string (never structural), and in a word whose bit is 0 there are no
    // backslashes and every ':' outside strings follows a closing quote.
    const uint32_t* odd = nullptr;
};

// kLineLong: run_line gave up on a whitespace skip longer than its skip
// bound (the caller evaluates the line again another way).
enum LineStatus : int { kLineDone = 0, kLineDeferred = 1, kLineLong = 2 };

GPJ_HD bool is_ws(uint8_t c) { return c == '\n' || c == '\r' || c == '\t' || c == ' '; }

// Every byte of x is one of the four whitespace bytes.
GPJ_HD bool all_ws32(uint32_t x) {
    return (eq_bytes(x, 0x20202020u) | eq_bytes(x, 0x0A0A0A0Au) | eq_bytes(x, 0x0D0D0D0Du) |
            eq_bytes(x, 0x09090909u)) == 0x80808080u;
}

// First position at or after j that is >= hi or not whitespace.  Short runs
// go byte by byte; a run longer than 32 bytes continues 32 aligned bytes per
// step (independent loads), so a skip over a long run of blanks does not
// wait for one memory round trip per byte.
template <typename P>
GPJ_HD P skip_ws(const uint8_t* file, P j, P hi) {
    for (int k = 0; k < 32; k++, ++j)
        if (j >= hi || !is_ws(file[j])) return j;
    for (; j < hi && (reinterpret_cast<uintptr_t>(file + j) & 7) != 0; ++j)
        if (!is_ws(file[j])) return j;
    for (; j + 32 <= hi; j += 32) {
        const uint32_t* w = reinterpret_cast<const uint32_t*>(file + j);
        uint32_t x[8];
#pragma unroll
        for (int i = 0; i < 8; i++) x[i] = w[i];
        bool all = true;
#pragma unroll
        for (int i = 0; i < 8; i++) all = all && all_ws32(x[i]);
        if (!all) break;
    }
    while (j < hi && is_ws(file[j])) ++j;
    return j;
}

// The bit helpers and the interpreter below are templates on the position
// type P: int64_t for positions in the file, int32_t for positions relative
// to a line's first word (run_line; half the integer work per step).

// A thread reads bitmaps K words at a time, words [K i, K i + K): the 32
// lanes of a warp are on 32 lines, so nearly every load waits for some lane's
// cache miss, and a search costs as many waits as it makes loads one after
// the other.  Two words for lines of a KB and more (2 GiB of 1.6 KB lines:
// 1031 us, 1206 with one word, 1057 with four), one for short lines, where
// the second is rarely wanted (256 MiB of 117-byte lines: 331 us, 373 with
// two).  Bitmaps given to the interpreter start on a 32-byte boundary at word
// 0 of their position type's base and are readable up to a multiple of four
// words.
template <int K>
struct Words {
    uint64_t w[K];
    GPJ_HD bool any() const {
        uint64_t x = 0;
#pragma unroll
        for (int i = 0; i < K; i++) x |= w[i];
        return x != 0;
    }
    // The first set bit's position, dropped (there is one).
    GPJ_HD int take() {
        int i = K - 1;
        uint64_t x = w[K - 1];
#pragma unroll
        for (int k = K - 2; k >= 0; k--) {
            i = w[k] ? k : i;
            x = w[k] ? w[k] : x;
        }
#pragma unroll
        for (int k = 0; k < K; k++) w[k] = k == i ? x & (x - 1) : w[k];
        return 64 * i + ctz64(x);
    }
    // without the words before word k and the bits of word k outside `mask`
    GPJ_HD void keep_from(int k, uint64_t mask) {
#pragma unroll
        for (int i = 0; i < K; i++) w[i] &= i < k ? 0ull : (i == k ? mask : ~0ull);
    }
};
// Words [chunk, chunk + K) (on the host none past `last`).
template <int K, typename P>
GPJ_HD Words<K> load_words(const uint64_t* bm, P chunk, P last) {
    static_assert(K == 1 || K == 2, "one load");
    Words<K> x;
#ifdef __CUDA_ARCH__
    (void)last;
    if constexpr (K == 2) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(bm + chunk);
        x.w[0] = a.x, x.w[1] = a.y;
    } else {
        x.w[0] = bm[chunk];
    }
#else
    for (int i = 0; i < K; i++) x.w[i] = chunk + i <= last ? bm[chunk + i] : 0;
#endif
    return x;
}

// First set bit of `bm` at a position in [from, limit), or `limit`.
template <int K, typename P>
GPJ_HD P next_bit(const uint64_t* bm, P from, P limit) {
    if (from >= limit) return limit;
    const P w = from >> 6, last = (limit - 1) >> 6;
    P c = w & ~static_cast<P>(K - 1);
    Words<K> x = load_words<K, P>(bm, c, last);
    x.keep_from(static_cast<int>(w - c), ~0ull << (from & 63));
    while (!x.any() && c + K <= last) {
        c += K;
        x = load_words<K, P>(bm, c, last);
    }
    const P p = x.any() ? (c << 6) + x.take() : limit;
    return p < limit ? p : limit;
}

// Last set bit of `bm` at a position in (floor, from], or -1; `first` is
// bm[from >> 6] (read only when from > floor).
template <typename P>
GPJ_HD P prev_bit(const uint64_t* bm, uint64_t first, P from, P floor) {
    if (from <= floor) return -1;
    P w = from >> 6;
    uint64_t m = first & (~0ull >> (63 - (from & 63)));
    for (;;) {
        if (m) {
            const P k = (w << 6) + 63 - clz64(m);
            return k > floor ? k : -1;
        }
        if ((w << 6) <= floor + 1) return -1;
        --w;
        m = bm[w];
    }
}

template <typename P>
GPJ_HD P prev_bit(const uint64_t* bm, P from, P floor) {
    return from <= floor ? -1 : prev_bit<P>(bm, bm[from >> 6], from, floor);
}

GPJ_HD uint32_t read_varint(const uint8_t* ir, int& pc) {
    uint32_t v = 0;
    int shift = 0;
    uint32_t b;
    while ((b = ir[pc++]) & 0x80u) {
        v |= (b & 0x7Fu) << shift;
        shift += 7;
    }
    return v | (b << shift);
}

// Per-level state of the interpreter: level_ends[k] (the end of the value
// entered at level k, -1 unknown) and current_index[k] (the array element
// counter, -1 before the array's '[' is reached).
//
// In registers/local memory, for every level a query may reach, in the
// interpreter's position type P.
template <typename P>
struct LocalLevelsT {
    P ends[kLevelSlots];
    P index[kLevelSlots];
    GPJ_HD void reset(P line_end) {
        ends[0] = line_end;
#pragma unroll
        for (int k = 1; k < kLevelSlots; k++) ends[k] = -1;
#pragma unroll
        for (int k = 0; k < kLevelSlots; k++) index[k] = -1;
    }
    GPJ_HD P end(int k) const { return ends[k]; }
    GPJ_HD void set_end(int k, P v) { ends[k] = v; }
    GPJ_HD P idx(int k) const { return index[k]; }
    GPJ_HD void set_idx(int k, P v) { index[k] = v; }
};
using LocalLevels = LocalLevelsT<int64_t>;

// In registers, for queries that go at most D - 1 levels down (a validated
// query's level is in [0, D) at every step): the arrays are only ever
// indexed by unrolled loops with constant indices, so they stay in
// registers; an access costs D selects instead of a local-memory round trip.
template <int D, typename P>
struct RegLevelsT {
    P ends[D];
    P index[D];
    GPJ_HD void reset(P line_end) {
        ends[0] = line_end;
#pragma unroll
        for (int k = 1; k < D; k++) ends[k] = -1;
#pragma unroll
        for (int k = 0; k < D; k++) index[k] = -1;
    }
    GPJ_HD P end(int k) const {
        P v = -1;
#pragma unroll
        for (int i = 0; i < D; i++) v = i == k ? ends[i] : v;
        return v;
    }
    GPJ_HD void set_end(int k, P v) {
#pragma unroll
        for (int i = 0; i < D; i++) ends[i] = i == k ? v : ends[i];
    }
    GPJ_HD P idx(int k) const {
        P v = -1;
#pragma unroll
        for (int i = 0; i < D; i++) v = i == k ? index[i] : v;
        return v;
    }
    GPJ_HD void set_idx(int k, P v) {
#pragma unroll
        for (int i = 0; i < D; i++) index[i] = i == k ? v : index[i];
    }
};

// Level slots a query needs: one more than its deepest level, rounded up to
// the register-state sizes the kernels are built for.
GPJ_HD int level_slots_for_depth(int depth) { return depth <= 4 ? 5 : (depth <= 8 ? 9 : kLevelSlots); }

// In caller-provided storage (e.g. shared memory, entries `stride` apart),
// as 32-bit offsets from the line start: for lines shorter than 2 GiB and
// queries no deeper than `slots - 1` levels.
struct PackedLevels {
    int32_t* ends;
    int32_t* index;
    int stride;
    int slots;
    int64_t origin;
    static constexpr int32_t kUnset = INT32_MIN;
    GPJ_HD void reset(int64_t line_end) {
        ends[0] = static_cast<int32_t>(line_end - origin);
        for (int k = 1; k < slots; k++) ends[k * stride] = kUnset;
        for (int k = 0; k < slots; k++) index[k * stride] = -1;
    }
    GPJ_HD int64_t end(int k) const {
        const int32_t v = ends[k * stride];
        return v == kUnset ? -1 : origin + v;
    }
    GPJ_HD void set_end(int k, int64_t v) { ends[k * stride] = v < 0 ? kUnset : static_cast<int32_t>(v - origin); }
    GPJ_HD int64_t idx(int k) const { return index[k * stride]; }
    GPJ_HD void set_idx(int k, int64_t v) { index[k * stride] = static_cast<int32_t>(v); }
};

// The four bytes at p, little endian (on the device two aligned loads, so
// up to three bytes after p + 4 are read as well).
GPJ_HD uint32_t load4(const uint8_t* p) {
#ifdef __CUDA_ARCH__
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    const uint32_t* w = reinterpret_cast<const uint32_t*>(a & ~static_cast<uintptr_t>(3));
    return __funnelshift_r(w[0], w[1], 8 * (a & 3));
#else
    return p[0] | p[1] << 8 | p[2] << 16 | static_cast<uint32_t>(p[3]) << 24;
#endif
}

// The key a MOVE_TO_KEY looks for, with the bytes that end right before the
// ':' of a match in the usual layout: the key's last three bytes (its opening
// quote among them when it is shorter) and its closing quote.  kWords: its
// bytes begin on a four-byte boundary.
constexpr int32_t kMaxSpan = 62;  // the quote `span` bytes before a ':' and the byte before it are at most a word back
template <bool kWords>
struct Key {
    const uint8_t* bytes;
    int32_t len;
    uint32_t tail, mask;  // mask 0: every candidate takes the general check
    int32_t span;         // from the key's opening quote to the ':', 0 where KeyScope::odd does not help
    GPJ_HD void set(const uint8_t* b, int32_t n) {
        bytes = b;
        len = n;
        bool quotes = false;
        for (int32_t i = 0; i < n && i <= kMaxSpan; i++) quotes = quotes || b[i] == '"';
        span = quotes || n + 2 > kMaxSpan ? 0 : n + 2;
        mask = n == 0 || b[n - 1] == '\\' ? 0u : (n == 1 ? 0xFFFFFF00u : ~0u);
        tail = 0x22000000u;
        if (n >= 1) tail |= static_cast<uint32_t>(b[n - 1]) << 16;
        if (n >= 1) tail |= static_cast<uint32_t>(n >= 2 ? b[n - 2] : '"') << 8;
        if (n >= 2) tail |= static_cast<uint32_t>(n >= 3 ? b[n - 3] : '"');
    }
    // The first n bytes are those at p (four more are readable with kWords).
    GPJ_HD bool starts(const uint8_t* p, int32_t n) const {
        bool same = true;
        if (kWords) {
            for (int32_t k = 0; same && k < n; k += 4)
                same = load4(p + k) == *reinterpret_cast<const uint32_t*>(bytes + k);
        } else {
            for (int32_t k = 0; same && k < n; k++) same = bytes[k] == p[k];
        }
        return same;
    }
};

// A query's instructions, one after the other: next() moves to the next one
// and returns its opcode; value, bytes and key() are its operands.  From the
// bytecode itself:
struct ByteCode {
    const uint8_t* ir;
    int pc = 0;
    uint32_t value = 0;
    const uint8_t* bytes = nullptr;
    GPJ_HD int next() {
        const int op = ir[pc++];
        if (op == 4 || op == 5 || op == 6) value = read_varint(ir, pc);
        if (op == 4 || op == 6) {
            bytes = ir + pc;
            pc += static_cast<int>(value);
        }
        return op;
    }
    GPJ_HD Key<false> key() const {
        Key<false> k;
        k.set(bytes, static_cast<int32_t>(value));
        return k;
    }
};

// From a program (query_program.h): 16-byte steps, then the keys' and
// strings' bytes.
struct ProgramStep {
    uint32_t op;     // opcode; Key::span << 8; Key::mask as 0, 1, 2 << 16
    uint32_t value;  // length or index
    uint32_t tail;   // Key::tail
    uint32_t at;     // the bytes, from the program's start
};
struct ProgramCode {
    const uint8_t* program;  // 16-byte aligned
    int pc = 0;
    uint32_t value = 0;
    const uint8_t* bytes = nullptr;
    uint32_t op = 0, tail = 0;
    GPJ_HD int next() {
#ifdef __CUDA_ARCH__
        const uint4 s = reinterpret_cast<const uint4*>(program)[pc++];
        op = s.x, value = s.y, tail = s.z, bytes = program + s.w;
#else
        const ProgramStep s = reinterpret_cast<const ProgramStep*>(program)[pc++];
        op = s.op, value = s.value, tail = s.tail, bytes = program + s.at;
#endif
        return op & 0xFF;
    }
    GPJ_HD Key<true> key() const {
        const uint32_t m = op >> 16;
        return Key<true>{bytes, static_cast<int32_t>(value), tail, m == 2 ? ~0u : (m ? 0xFFFFFF00u : 0u),
                         static_cast<int32_t>((op >> 8) & 0xFF)};
    }
};
GPJ_HD ByteCode code_of(const uint8_t* ir) { return ByteCode{ir}; }
GPJ_HD ProgramCode code_of(const ProgramCode& p) { return p; }

// What a key search looks at.
template <typename P>
struct KeyScope {
    const uint8_t* file;
    P hi;  // bytes at or after it are not read
    const uint64_t* string_index;
    P line_start;
    // LineView::odd, and the number there of the word at position 0
    const uint32_t* odd;
    uint32_t odd_base;
    // Of the 32 words of entry i: bit k set when word k or the one before it is odd.
    GPJ_HD uint32_t odd_or_after(uint32_t i) const {
        const uint32_t x = odd[i];
        return x | (x << 1) | (i ? odd[i - 1] >> 31 : 0u);
    }
};

// Of the structural ':' `x` of a word, those of keys whose opening quote is
// `span` bytes before them (`marks`: the word of LineView::colon with odd,
// `before` the one before it).
GPJ_HD uint64_t of_length(uint64_t x, uint64_t marks, uint64_t before, int32_t span) {
    return x & ((marks << span) | (before >> (64 - span)));
}

// The key candidates among the structural ':' of a chunk (`x`: a level's
// bitmap): `marks` is the chunk of LineView::colon (with odd), `before` the
// word before it, bit i of `odd` set where word i or the one before it is
// odd.  Elsewhere each ':' follows a closing quote and the quotes before it
// are not escaped, so a key without quotes matches only where its opening
// quote is `span` bytes before the ':': all candidates are judged at once, by
// their keys' lengths, and the file's bytes are read for the few that remain.
template <int K>
GPJ_HD void of_length(Words<K>& x, const Words<K>& marks, uint64_t before, uint32_t odd, int32_t span) {
#pragma unroll
    for (int i = 0; i < K; i++) {
        x.w[i] &= marks.w[i];
        if (!((odd >> i) & 1u)) x.w[i] = of_length(x.w[i], marks.w[i], i ? marks.w[i - 1] : before, span);
    }
}

// Whether the string before the structural ':' at p is the key
// (find_value.cu:225-251): the key's bytes end at the last in-string byte
// before p, with a '"' before them.
//
// A '"' right before p that no backslash precedes closes a string (the ':'
// is outside strings), so that byte is p - 2 and the file's bytes alone
// decide: one four-byte comparison rejects nearly every other key, without
// the string index and the key's bytes one by one.  Anything else (blanks
// before the ':', a backslash, the line's or view's edges, a key with mask
// 0) takes the general check.
template <typename P, bool kWords>
GPJ_HD bool key_at(const KeyScope<P>& v, const Key<kWords>& key, P p) {
    if (key.mask != 0 && p - v.line_start >= 4 && p + 4 <= v.hi) {
        const uint32_t t = load4(v.file + p - 4);
        if (((t ^ key.tail) & key.mask) == 0) {
            const int64_t start = static_cast<int64_t>(p) - 2 - key.len;
            return key.len <= 2 ||
                   (start >= v.line_start && v.file[start] == '"' && key.starts(v.file + start + 1, key.len - 3));
        }
        if ((t & 0xFF000000u) == 0x22000000u && (t & 0x00FF0000u) != 0x005C0000u) return false;
    }
    const int64_t start = static_cast<int64_t>(prev_bit<P>(v.string_index, p - 1, v.line_start)) - key.len;
    bool same = start >= v.line_start && v.file[start] == '"';
    for (int32_t k = 0; same && k < key.len; k++) same = key.bytes[k] == v.file[start + 1 + k];
    return same;
}

// How the interpreter scans: one thread alone (SeqScanOf), or the 32 lanes of
// a warp together on one line (WarpScan, query_kernel.cu), every lane
// holding the same interpreter state.
template <int K>
struct SeqScanOf {
    template <typename P>
    GPJ_HD static P next(const uint64_t* bm, P from, P limit) {
        return next_bit<K, P>(bm, from, limit);
    }
    // First structural ':' of `bits` in [from, limit) whose string is the key, or `limit`.
    template <typename P, bool kWords>
    GPJ_HD static P find_key(const KeyScope<P>& v, const Key<kWords>& key, const uint64_t* bits, const uint64_t* colon, P from,
                             P limit) {
        if (from >= limit) return limit;
        const P w = from >> 6, last = (limit - 1) >> 6;
        P c = w & ~static_cast<P>(K - 1);
        // Each lane of a warp runs the inner loop to its next candidate, then
        // the candidates are checked together (and each loop has one exit, so
        // that the lanes meet again).
        const bool by_length = v.odd && key.span;
        uint32_t number = v.odd_base + static_cast<uint32_t>(c);  // the chunk's first word in the file
        uint64_t before = by_length && number ? colon[c - 1] : 0;
        auto load = [&]() -> Words<K> {
            Words<K> x = load_words<K, P>(bits, c, last);
            if (colon) {
                const Words<K> m = load_words<K, P>(colon, c, last);
                of_length(x, m, before, by_length ? v.odd_or_after(number >> 5) >> (number & 31) : ~0u, key.span);
                before = m.w[K - 1];
            }
            return x;
        };
        Words<K> x = load();
        x.keep_from(static_cast<int>(w - c), ~0ull << (from & 63));
        P hit = -1;
        while (hit < 0) {
            while (!x.any() && c + K <= last) {
                c += K;
                number += K;
                x = load();
            }
            if (!x.any()) break;
            const P p = (c << 6) + x.take();
            if (p >= limit || ((colon || v.file[p] == ':') && key_at<P>(v, key, p))) hit = p;
        }
        return hit >= 0 && hit < limit ? hit : limit;
    }
    // Position of the `count`-th (from 1) ',' among the bytes of `bits` in [from, limit), or `limit`.
    template <typename P>
    GPJ_HD static P find_comma(const uint8_t* file, const uint64_t* bits, const uint64_t* colon, P from, P limit,
                               int64_t count) {
        if (from >= limit || count < 1) return limit;
        const P w = from >> 6, last = (limit - 1) >> 6;
        P c = w & ~static_cast<P>(K - 1);
        auto load = [&]() -> Words<K> {
            Words<K> x = load_words<K, P>(bits, c, last);
            if (colon) {
                const Words<K> m = load_words<K, P>(colon, c, last);
#pragma unroll
                for (int i = 0; i < K; i++) x.w[i] &= ~m.w[i];
            }
            return x;
        };
        Words<K> x = load();
        x.keep_from(static_cast<int>(w - c), ~0ull << (from & 63));
        P hit = -1;
        while (hit < 0) {
            while (!x.any() && c + K <= last) {
                c += K;
                x = load();
            }
            if (!x.any()) break;
            const P p = (c << 6) + x.take();
            if (p >= limit || (file[p] == ',' && --count == 0)) hit = p;
        }
        return hit >= 0 && hit < limit ? hit : limit;
    }
    template <typename P>
    GPJ_HD static P skip(const uint8_t* file, P j, P hi) {
        return skip_ws<P>(file, j, hi);
    }
    GPJ_HD static void store(int64_t* res, int64_t k, int64_t v) { res[k] = v; }
};
using SeqScan = SeqScanOf<2>;

// Runs the validated query `code` (ByteCode, ProgramCode) on the line [line_start, line_end) and writes
// (start, end) pairs to res[2*k], res[2*k+1] for the k-th STORE_RESULT.
// res must hold -1 on entry.  Returns kLineDeferred when the view ends
// before the line's evaluation does (`skip_end`: what a whitespace skip that
// reaches `hi` returns).  Positions are of type P and relative to `base`
// (added to the stored results); `file`, `string_index`, `levels` and
// `colon` are rebased to match (`odd` is not).  `lv` holds the per-level state.
template <typename P, typename Levels, typename Scan, typename Code>
GPJ_HD int run_line_core(const uint8_t* file, P n, P hi, int skip_end, const uint64_t* string_index,
                         const uint64_t* levels, int64_t level_size, const uint64_t* colon, const uint32_t* odd,
                         P line_start, P line_end, Code code, int64_t* res, int64_t base, Levels& lv,
                         int& stored) {
    lv.reset(line_end);

    int cur = 0, result_index = 0;
    stored = 0;
    const KeyScope<P> scope{file, hi, string_index, line_start, odd, static_cast<uint32_t>(base >> 6)};
    int64_t want_index = -1;
    P j = line_start;
    // The end of the value entered at level cur (-1: none found).  The levels
    // above keep theirs in lv while the query is below them: MOVE_UP forgets
    // the end of the level it leaves, so MOVE_DOWN always looks for a new one.
    P cend = line_end;
    while (j < cend && j < n) {
        // The opcodes up to the next search.
        bool to_key = false, to_index = false;
        while (!to_key && !to_index) {
            switch (code.next()) {
                case 0:  // END
                    return kLineDone;
                case 1: {  // STORE_RESULT (find_value.cu:59-82)
                    j = Scan::template skip<P>(file, j, hi);  // [bounded] stops at end of file
                    if (j >= hi && skip_end) return kLineDeferred;
                    Scan::store(res, 2 * result_index, base + j);
                    Scan::store(res, 2 * result_index + 1, cend < 0 ? -1 : base + cend);
                    stored = ++result_index;
                    break;
                }
                case 2:  // MOVE_UP (:83-90)
                    if (cend < 0) return kLineDone;  // [bounded] would continue at j=-1
                    j = cend;
                    cend = lv.end(--cur);
                    break;
                case 3: {  // MOVE_DOWN (:91-111): end of the value = next structural one level up
                    const P m = Scan::template next<P>(levels + level_size * cur, j + 1, cend);
                    lv.set_end(cur++, cend);
                    cend = m < cend ? m : -1;
                    break;
                }
                case 4:  // MOVE_TO_KEY (:112-130)
                    to_key = true;
                    break;
                case 5:  // MOVE_TO_INDEX (:131-169)
                    want_index = code.value;
                    if (lv.idx(cur) == -1) {
                        j = Scan::template skip<P>(file, j, hi);  // [bounded] only whitespace may precede '['
                        if (j >= hi) return skip_end;
                        if (file[j] != '[') return kLineDone;
                        lv.set_idx(cur, 0);
                    }
                    if (want_index == 0)
                        ++j;
                    else
                        to_index = true;
                    break;
                case 6: {  // EXPRESSION_STRING_EQUALS (:170-210)
                    const P len = static_cast<P>(code.value);
                    const uint8_t* want = code.bytes;
                    j = Scan::template skip<P>(file, j, hi);  // [bounded]
                    if (j >= hi && skip_end) return kLineDeferred;
                    if (cend - j != len) return kLineDone;
                    for (P k = 0; k < len; k++)
                        if (want[k] != file[j + k]) return kLineDone;
                    break;
                }
                default:
                    return kLineDone;
            }
        }
        // The search, among the structural bytes of the current level (nothing
        // happens at any other byte): a ':' whose key matches (:225-251), or
        // the ',' before the wanted element (:252-259).  A search that fails
        // ends the line.
        const P lim = cend < n ? cend : n;
        const uint64_t* bits = levels + level_size * cur;
        if (to_key) {
            j = Scan::find_key(scope, code.key(), bits, colon, j, lim);
        } else {
            j = Scan::template find_comma<P>(file, bits, colon, j, lim, want_index - lv.idx(cur));
            lv.set_idx(cur, static_cast<P>(want_index));
        }
        if (j >= lim) return kLineDone;
        ++j;
    }
    return kLineDone;
}

// The interpreter on a view's positions as they are (64-bit), with the
// per-level state in `lv` (LocalLevels, PackedLevels); res must hold -1 on
// entry (only the stored results are written).
template <typename Levels>
GPJ_HD int run_line_with(const LineView& v, int64_t line_start, int64_t line_end, const uint8_t* ir,
                         int64_t* res, Levels& lv) {
    int stored = 0;
    return run_line_core<int64_t, Levels, SeqScan>(v.file, v.n, v.hi, v.hi < v.n ? kLineDeferred : kLineDone, v.string_index,
                                  v.levels, v.level_size, v.colon, v.odd, line_start, line_end, code_of(ir), res, 0, lv,
                                  stored);
}

// Largest line-relative position the 32-bit interpreter handles.
constexpr int64_t kRelLimit = (1ll << 31) - 4096;

// The interpreter in 64-bit positions with the level state in local memory,
// for lines the 32-bit form cannot hold; a separate function, so that its
// state does not add to the registers of the 32-bit form's caller.  Writes
// every one of the res_len entries once.
template <typename Scan = SeqScan, typename Ir>
#ifdef __CUDACC__
static __host__ __device__ __noinline__
#else
static __attribute__((noinline))
#endif
int run_line_wide(const LineView& v, int64_t line_start, int64_t line_end, Ir ir, int64_t* res,
                  int64_t res_len) {
    LocalLevels lv;
    int stored = 0;
    const int r = run_line_core<int64_t, LocalLevels, Scan>(v.file, v.n, v.hi, v.hi < v.n ? kLineDeferred : kLineDone,
                                                            v.string_index, v.levels, v.level_size, v.colon, v.odd,
                                                            line_start, line_end, code_of(ir), res, 0, lv, stored);
    for (int64_t k = 2 * static_cast<int64_t>(stored); k < res_len; k++) Scan::store(res, k, -1);
    return r;
}

// run_line_with with positions relative to the line's first four words
// in 32 bits (the usual case: half the integer work per step) and the
// per-level state in registers for queries whose level stays below D.
// Every one of the res_len entries is written once: the stored results,
// then -1 for the slots the line did not reach (res need not be
// initialised).  Lines whose end lies more than rel_limit (<= kRelLimit)
// bytes past their start run in 64 bits; a whitespace skip that reaches
// rel_limit (bytes past it exist) stops there and the line is evaluated
// again in 64 bits.  With a skip_bound, a whitespace skip that runs more
// than skip_bound bytes past the line's end (into the blank lines after it)
// stops there too and run_line returns kLineLong, with res partly written,
// for the caller to evaluate the line again (by a warp, query_kernel.cu).
template <int D = kLevelSlots, typename Scan = SeqScan, typename Ir>
GPJ_HD int run_line(const LineView& v, int64_t line_start, int64_t line_end, Ir ir, int64_t* res,
                    int64_t res_len, int64_t rel_limit = kRelLimit, int64_t skip_bound = -1) {
    const int64_t base = line_start & ~static_cast<int64_t>(255);
    int stored = 0;
    if (line_end - base <= rel_limit) {
        const int64_t lim =
            skip_bound >= 0 && line_end - base + skip_bound < rel_limit ? line_end - base + skip_bound : rel_limit;
        const bool clamped = v.hi - base > lim;
        const int32_t hi = static_cast<int32_t>(clamped ? lim : v.hi - base);
        const int32_t n = static_cast<int32_t>(v.n - base > rel_limit ? rel_limit : v.n - base);
        const int skip_end = clamped || v.hi < v.n ? kLineDeferred : kLineDone;
        const int64_t w = base >> 6;
        RegLevelsT<D, int32_t> lv;
        const int r = run_line_core<int32_t, RegLevelsT<D, int32_t>, Scan>(
            v.file + base, n, hi, skip_end, v.string_index + w, v.levels + w, v.level_size,
            v.colon ? v.colon + w : nullptr, v.odd, static_cast<int32_t>(line_start - base),
            static_cast<int32_t>(line_end - base), code_of(ir), res, base, lv, stored);
        if (r != kLineDeferred || !clamped) {
            for (int64_t k = 2 * static_cast<int64_t>(stored); k < res_len; k++) Scan::store(res, k, -1);
            return r;
        }
        if (skip_bound >= 0) return kLineLong;
    }
    return run_line_wide<Scan>(v, line_start, line_end, ir, res, res_len);
}

// Deepest level a validated query's bytecode reaches (its MOVE_DOWNs).
GPJ_HD int bytecode_depth(const uint8_t* ir) {
    int pc = 0, level = 0, deepest = 0;
    for (;;) {
        const uint8_t op = ir[pc++];
        if (op == 0 || op > 6) return deepest;
        if (op == 2) --level;
        if (op == 3 && ++level > deepest) deepest = level;
        if (op == 4 || op == 6) {
            const uint32_t len = read_varint(ir, pc);
            pc += static_cast<int>(len);
        }
        if (op == 5) read_varint(ir, pc);
    }
}

// run_line with the register state sized for queries no deeper than `depth`
// (the sizes the kernels are instantiated for).
template <typename Ir>
GPJ_HD int run_line_depth(int depth, const LineView& v, int64_t line_start, int64_t line_end, Ir ir,
                          int64_t* res, int64_t res_len, int64_t rel_limit = kRelLimit, int64_t skip_bound = -1) {
    switch (level_slots_for_depth(depth)) {
        case 5:
            return run_line<5>(v, line_start, line_end, ir, res, res_len, rel_limit, skip_bound);
        case 9:
            return run_line<9>(v, line_start, line_end, ir, res, res_len, rel_limit, skip_bound);
        default:
            return run_line<kLevelSlots>(v, line_start, line_end, ir, res, res_len, rel_limit, skip_bound);
    }
}

}  // namespace gpj
