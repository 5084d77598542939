// Device memory of a file's index, as it is first allocated.
#pragma once

#include <algorithm>
#include <cstdint>

namespace gpj {

// Words allocated for one bitmap of n bytes: find_value reads whole aligned
// groups of words, and every bitmap begins on a 128-byte boundary.
inline int64_t bitmap_words(int64_t n) { return ((n + 63) / 64 + 15) / 16 * 16; }

// 64-bit words of IndexParams::odd.
inline int64_t odd_words(int64_t n) { return ((n + 63) / 64 + 63) / 64; }

// Lines there is room for at first: one in 256 bytes and 1024, less what the
// odd words and the bitmaps' ends take, so that an index with that many
// levels is no larger than its bitmaps' words and that many lines (what the
// server counts for a resident corpus).
inline int64_t first_lines(int64_t n, int levels) {
    const int64_t ends = (2 + levels) * (bitmap_words(n) - (n + 63) / 64);
    return std::min<int64_t>(n + 1, n / 256 + 1024 - odd_words(n) - ends);
}

// Words of the whole index: string index, key marks, levels, newlines, odd words.
inline int64_t index_words(int64_t n, int levels) {
    return (2 + levels) * bitmap_words(n) + first_lines(n, levels) + odd_words(n);
}

}  // namespace gpj
