// Host-side interface of the find_value kernel (query_kernel.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "query_items.cuh"

namespace gpj {

// A (line, query) item handed from the thread-per-line kernels to the
// warp-per-line kernel (line of file `file` of the launch).
struct LongItem {
    int64_t line;
    int32_t file;
    int32_t query;
};

// Where the thread-per-line kernels put lines longer than `bytes`, which a
// whole warp then evaluates (find_value_warp_kernel): `items` holds `cap` entries,
// `count` (zeroed before the launch) counts them; items past `cap` are
// evaluated by their thread.  items == nullptr: no line is handed over.
struct LongLines {
    LongItem* items;
    unsigned long long* count;
    int64_t cap;
    int64_t bytes;
};

// Threads per CTA of find_value_kernel and find_value_batch_kernel (a
// multiple of 32; grids are sized in these CTAs), and the CTAs per SM their
// register budget is set for, by register-state size D: 7 (at most 72
// registers) for D = 5, 5 for D = 9 (32 paths over 64 MiB: 309 us, 340 with
// 6), 4 for D = 17.  Threads wait for their lines' cache misses, more of them
// spill: 8 CTAs for D = 5 took 1001 us at 2 GiB of tweets where 7 take 1031,
// but 153 and 78 us at 256 and 64 MiB where they take 155 and 76.
constexpr int kQueryThreads = 128;
template <int D>
constexpr int kQueryMinCtas = D <= 5 ? 7 : (D <= 9 ? 5 : 4);
// The same for the warp-per-line kernels, and the CTAs per SM they launch
// for the handed-over lines (whose number the host does not know).
constexpr int kWarpThreads = 64;
template <int D>
constexpr int kWarpMinCtas = D <= 5 ? 12 : (D <= 9 ? 10 : 8);
constexpr int kListCtasPerSm = 8;

struct QueryParams {
    const uint8_t* file;
    int64_t n;
    const int64_t* newlines;
    int64_t num_lines;
    const uint64_t* string_index;
    const uint64_t* leveled;
    int64_t level_size;       // words between levels, a multiple of 4 (LineView)
    const uint8_t* programs;  // all queries' programs (query_program.h)
    const int32_t* offsets;   // start of query q's there, a multiple of 16
    int num_queries;
    int slots;     // result slots per line (max num_results)
    int64_t* out;       // [num_queries][out_lines][slots][2]
    int64_t out_lines;  // query stride of `out` (>= num_lines)
    // Optional, for a file still being indexed: only lines [range[0],
    // range[1]) (device memory, read by the kernel), whose newline-index
    // entries up to range[1] are written; the last of them ends at the file
    // end when `last`, else at newlines[range[1]].  Lines whose results or
    // end do not fit out_lines / newline_cap are skipped (the caller sees the
    // line count and evaluates again).
    const int64_t* range;
    int last;
    int64_t newline_cap;
    // Bytes at or after `hi` are not read (n: all may be; else, with `range`,
    // they are still on their way to the device): a query whose whitespace
    // skip gets there sets kErrDeferred in status[1], its results are not valid.
    int64_t hi;
    unsigned long long* status;
    // Optional (both or none), IndexParams::marks and odd: key searches jump
    // between the ':' of keys of the right length, index searches between the
    // other structural bytes.
    const uint64_t* marks;
    const uint32_t* odd;
    // deepest level of the launch's queries (sizes the interpreter's
    // register state)
    int depth;
    // every line by a warp (query_by_warp; not with `range`): one launch of
    // the warp-per-line kernel alone
    bool by_warp;
    // a thread reads one bitmap word at a time instead of two
    bool short_lines;
    LongLines long_lines;
};

// find_value over the launch's lines: a thread per (line, query) with `grid`
// CTAs, then (when p.long_lines.items is set) the long lines a warp each with
// `warp_grid` CTAs; or, by_warp, all lines a warp each.
cudaError_t launch_find_value(const QueryParams& p, int grid, int warp_grid, cudaStream_t stream);
// Resident CTAs per SM of the find_value kernel for queries of that depth.
int find_value_max_ctas_per_sm(int depth);

// One file of a batched find_value launch: its index, its queries and where
// their results go ([num_queries][out_lines][slots][2]); its lines are
// [line_begin, line_begin + num_lines) of the batch's line numbering.
struct QueryFile {
    const uint8_t* file;
    int64_t n;
    const int64_t* newlines;
    int64_t num_lines;
    const uint64_t* string_index;
    const uint64_t* leveled;
    int64_t level_size;
    const uint8_t* programs;
    const int32_t* offsets;
    int num_queries;
    int slots;
    int64_t* out;
    int64_t out_lines;
    // first of the file's items in the batch's thread-per-line launch:
    // ceil(num_lines / 32) blocks of 32 lines x num_queries (a multiple of 32,
    // so no warp spans two files), none for a file whose lines get a warp each
    int64_t item_begin;
    const uint64_t* marks;  // optional, as in QueryParams
    const uint32_t* odd;
    // first of its (line, query) pairs in the warp-per-line launch (none for
    // the other files)
    int64_t warp_begin;
};

// Every (line, query) item of every file of the batch (`files`: device
// array, ascending item_begin and warp_begin; `items` thread and `warp_items`
// warp items in all; `depth` the deepest level of any of their queries).  A
// thread-per-line warp's lanes run one query on 32 lines of one file, and the
// warps of a block of lines run its queries side by side.
cudaError_t launch_find_value_batch(const QueryFile* files, int nfiles, int64_t items, int64_t warp_items, int depth,
                                    const LongLines& long_lines, int grid, int warp_grid, cudaStream_t stream);

}  // namespace gpj
