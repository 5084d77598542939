// Work distribution of the find_value kernels (query_kernel.cu): which
// (line, query) pair a grid-stride item number stands for.  __host__
// __device__ so the test suite can check on the CPU that every pair is
// visited exactly once.
#pragma once

#include <cstdint>

#include "word_ops.cuh"

namespace gpj {

// Mean line length from which every line of a file gets a warp (1 GiB with
// lines of 100 B-1 MiB, 27,000 pairs: 207 us, against 870 with a thread for
// each line up to 64 KiB; 1.6 KB lines are the threads').
constexpr int64_t kWarpLineBytes = 4096;

// A file's lines are taken in blocks of 32; block b owns the items
// [item_begin + b * group, item_begin + (b + 1) * group), group = 32 *
// num_queries: one warp per query, one line per lane, so a warp's lanes
// follow one opcode sequence and the block's queries run side by side on
// one SM over the same lines.  The queries of block b are rotated by the
// grid-stride round its first item falls in (the same for all of the
// block's warps), so a warp meets a different query in each round and a
// cheap query does not leave it idle.  `stride` = threads of the grid (a
// multiple of 32); `k` = item number within the file.  Returns false for
// the padding items past the last line.
GPJ_HD bool query_item(int64_t k, int64_t item_begin, int64_t num_lines, int num_queries, int64_t stride,
                       int64_t* line, int* query) {
    const int64_t group = 32 * static_cast<int64_t>(num_queries);
    if (item_begin + k < INT32_MAX && stride < INT32_MAX) {
        // (three divisions an item, several times cheaper in 32 bits)
        const uint32_t g = static_cast<uint32_t>(group), b = static_cast<uint32_t>(k) / g;
        const uint32_t r = static_cast<uint32_t>(k) - b * g;
        const uint32_t round = (static_cast<uint32_t>(item_begin) + b * g) / static_cast<uint32_t>(stride);
        *query = static_cast<int>(((r >> 5) + round) % static_cast<uint32_t>(num_queries));
        *line = (static_cast<int64_t>(b) << 5) + (r & 31);
        return *line < num_lines;
    }
    const int64_t b = k / group;
    const int64_t r = k - b * group;
    *query = static_cast<int>(((r >> 5) + (item_begin + b * group) / stride) % num_queries);
    *line = (b << 5) + (r & 31);
    return *line < num_lines;
}

// Items of a file: ceil(num_lines / 32) blocks of 32 * num_queries (a
// multiple of 32, so no warp spans two files of a batch).
GPJ_HD int64_t query_items(int64_t num_lines, int num_queries) {
    return (num_lines + 31) / 32 * 32 * num_queries;
}

// Whether a file of `lines` lines and `bytes` bytes has each (line, query)
// pair evaluated by a warp instead of a thread: where lines are long, or
// there are few pairs (`few`: as many as finish sooner that way).
GPJ_HD bool query_by_warp(int64_t lines, int64_t bytes, int num_queries, int64_t few) {
    return lines * num_queries <= few || bytes / kWarpLineBytes >= lines;
}

// Mean line length under which a thread reads one bitmap word at a time
// (Words, interp.cuh: a line of under four words rarely wants the next).  Only
// for a whole file: the files of a batch's launch differ in their lines, and a
// chunk's lines are not counted when its queries are launched.
constexpr int64_t kShortLineBytes = 256;

}  // namespace gpj
