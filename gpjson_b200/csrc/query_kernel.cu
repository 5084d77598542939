// find_value: the per-line JSONPath interpreter kernel on sm_100a.
//
// The reference launches find_value once per query with 512x1024 threads
// and a contiguous range of lines per thread
// (functions/QueryFunction.java:201-241, kernels/find_value.cu:12-23).
// Here one launch evaluates every query of the call.  Lines are taken in
// blocks of 32; a block's (line, query) items are nq warps, one query per
// warp and one line per lane, so a warp's lanes follow the same opcode
// sequence and the block's queries run side by side on one SM: the lines'
// bitmap words and key bytes come from DRAM once and are re-read from L1/L2
// by the other queries' warps while still there.  Warps stride over the
// blocks (grid sized to the SMs) and rotate through the queries from one
// block to the next, so a cheap query does not leave its warp idle.  Each
// query writes its own slots, so its results equal a solo run.
//
// Long lines, and all lines where there are few (query_by_warp), get a warp
// each in a second kernel: its searches look at 2 KiB of bitmap per step.
//
// Bound by the waits for cache misses (long scoreboard 7 of 13 stall cycles
// per instruction; DRAM 2.3 TB/s, ALU 50 %).  256 MiB of tweets, 4 queries:
// 145 us and 70 M warp instructions; 271 us and 127 M when every key
// candidate was checked byte by byte, 197 us and 76 M when each cost a load
// of the file's bytes before it, before candidates were judged by their
// keys' lengths (KeyScope) and the queries decoded on the host
// (query_program.h).
#include <cstdint>

#include "device_common.cuh"
#include "interp.cuh"
#include "query_items.cuh"
#include "query_kernel.h"

namespace gpj {

namespace {

// The scans of one line by the 32 lanes of a warp together (all lanes call
// with the same arguments and hold the same interpreter state): a search
// for the next structural bit, a key or an array element reads 32 to 256
// bitmap words per step, a whitespace skip 512 bytes, so a line of a megabyte costs
// its warp a few hundred dependent memory round trips instead of one lane
// tens of thousands.
struct WarpScan {
    // A search walks its words 32 at a time, one to a lane; beyond the first
    // 32 it loads kWide x 32 per step (independent loads) and looks at them
    // only when one holds a candidate.
    static constexpr int kWide = 8;
    // Calls use(first word, this lane's word) for 32 words after 32, without
    // the bytes before `from` and at or after `limit` (`filt` keeps or, with
    // flip = ~0, drops its bytes), until it returns a position >= 0, which is
    // returned, or the words end (limit).  Words of zeros are not passed on.
    template <typename P, typename Use>
    __device__ static P walk(const uint64_t* bits, const uint64_t* filt, uint64_t flip, P from, P limit, Use use) {
        if (from >= limit) return limit;
        const int lane = threadIdx.x & 31;
        const P last = (limit - 1) >> 6;
        auto word = [&](P i) -> uint64_t { return bits[i] & (filt ? filt[i] ^ flip : ~0ull); };
        auto word_or_none = [&](P i) -> uint64_t {
            if (i > last) return 0;
            const uint64_t x = word(i);
            return i == last ? x & (~0ull >> (63 - ((limit - 1) & 63))) : x;
        };
        P w = from >> 6;
        uint64_t x0 = word_or_none(w + lane);
        if (lane == 0) x0 &= ~0ull << (from & 63);
        if (__any_sync(~0u, x0 != 0)) {
            const P p = use(w, x0);
            if (p >= 0) return p;
        }
        for (w += 32; w <= last; w += 32 * kWide) {
            uint64_t x[kWide];
            if (w + 32 * kWide <= last) {
#pragma unroll
                for (int u = 0; u < kWide; u++) x[u] = word(w + 32 * u + lane);
            } else {
#pragma unroll
                for (int u = 0; u < kWide; u++) x[u] = word_or_none(w + 32 * u + lane);
            }
            uint64_t any = 0;
#pragma unroll
            for (int u = 0; u < kWide; u++) any |= x[u];
            if (!__any_sync(~0u, any != 0)) continue;
            // (one copy of `use`: the words are picked by selects)
#pragma unroll 1
            for (int u = 0; u < kWide; u++) {
                uint64_t xu = x[0];
#pragma unroll
                for (int i = 1; i < kWide; i++) xu = u == i ? x[i] : xu;
                if (!__any_sync(~0u, xu != 0)) continue;
                const P p = use(w + 32 * u, xu);
                if (p >= 0) return p;
            }
        }
        return limit;
    }
    template <typename P>
    __device__ static P next(const uint64_t* bm, P from, P limit) {
        return walk<P>(bm, nullptr, 0, from, limit, [](P w, uint64_t x) -> P {
            const unsigned hit = __ballot_sync(~0u, x != 0);
            const int f = __ffs(static_cast<int>(hit)) - 1;
            return ((w + f) << 6) + ctz64(__shfl_sync(~0u, x, f));
        });
    }
    // each lane checks the candidates of its own word
    template <typename P, bool kWords>
    __device__ static P find_key(const KeyScope<P>& v, const Key<kWords>& key, const uint64_t* bits, const uint64_t* colon,
                                 P from, P limit) {
        return walk<P>(bits, colon, 0, from, limit, [&](P w, uint64_t x) -> P {
            P found = -1;
            for (; x && found < 0; x &= x - 1) {
                const P p = ((w + (threadIdx.x & 31)) << 6) + ctz64(x);
                if ((colon || v.file[p] == ':') && key_at<P>(v, key, p)) found = p;
            }
            const unsigned hit = __ballot_sync(~0u, found >= 0);
            return hit ? __shfl_sync(~0u, found, __ffs(static_cast<int>(hit)) - 1) : -1;
        });
    }
    // each lane counts the ',' of its own word
    template <typename P>
    __device__ static P find_comma(const uint8_t* file, const uint64_t* bits, const uint64_t* colon, P from, P limit,
                                   int64_t count) {
        if (count < 1) return limit;
        return walk<P>(bits, colon, ~0ull, from, limit, [&](P w, uint64_t x) -> P {
            const int lane = threadIdx.x & 31;
            uint64_t commas = 0;
            for (; x; x &= x - 1)
                if (file[((w + lane) << 6) + ctz64(x)] == ',') commas |= x & (~x + 1);
            if (!__any_sync(~0u, commas != 0)) return -1;
            int incl = popc64(commas);
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const int o = __shfl_up_sync(~0u, incl, off);
                if (lane >= off) incl += o;
            }
            const unsigned reached = __ballot_sync(~0u, incl >= count);
            if (reached) {
                const int f = __ffs(static_cast<int>(reached)) - 1;
                const int before = __shfl_sync(~0u, incl, f > 0 ? f - 1 : 0);
                uint64_t m = __shfl_sync(~0u, commas, f);
                for (int64_t skip = count - 1 - (f > 0 ? before : 0); skip > 0; skip--) m &= m - 1;
                return ((w + f) << 6) + ctz64(m);
            }
            count -= __shfl_sync(~0u, incl, 31);
            return -1;
        });
    }
    // first position at or after j that is >= hi or not whitespace
    template <typename P>
    __device__ static P skip(const uint8_t* file, P j, P hi) {
        const int lane = threadIdx.x & 31;
        for (int k = 0; k < 32; k++, ++j)
            if (j >= hi || !is_ws(file[j])) return j;
        for (; j < hi && (reinterpret_cast<uintptr_t>(file + j) & 15) != 0; ++j)
            if (!is_ws(file[j])) return j;
        for (;; j += 512) {
            const P q = j + 16 * lane;
            P stop = -1;  // this lane's answer among its 16 bytes, if any
            if (q + 16 <= hi) {
                const uint4 v = *reinterpret_cast<const uint4*>(file + q);
                if (!(all_ws32(v.x) && all_ws32(v.y) && all_ws32(v.z) && all_ws32(v.w))) {
                    for (int b = 0; b < 16; b++) {
                        if (!is_ws(file[q + b])) {
                            stop = q + b;
                            break;
                        }
                    }
                }
            } else {
                for (int b = 0; b < 16; b++) {
                    const P r = q + b;
                    if (r >= hi || !is_ws(file[r])) {
                        stop = r;
                        break;
                    }
                }
            }
            const unsigned hit = __ballot_sync(~0u, stop >= 0);
            if (hit) return __shfl_sync(~0u, stop, __ffs(static_cast<int>(hit)) - 1);
        }
    }
    __device__ static void store(int64_t* res, int64_t k, int64_t v) {
        if ((threadIdx.x & 31) == 0) res[k] = v;
    }
};

// Hands item (line, file, query) to the warp-per-line kernel; false when the
// list is full (the caller evaluates it).
__device__ __forceinline__ bool hand_over(const LongLines& L, int64_t line, int file, int query) {
    const unsigned long long slot = atomicAdd(L.count, 1ull);
    if (static_cast<int64_t>(slot) >= L.cap) return false;
    L.items[slot] = LongItem{line, file, query};
    return true;
}

__device__ __forceinline__ int64_t handed_over(const LongLines& L) {
    if (!L.items) return 0;
    const unsigned long long count = *L.count;
    return count < static_cast<unsigned long long>(L.cap) ? static_cast<int64_t>(count) : L.cap;
}

// D: level slots of the interpreter's register state (level_slots_for_depth
// of the deepest query of the launch); K: bitmap words read at a time.
template <int D, int K>
__global__ void __launch_bounds__(kQueryThreads, kQueryMinCtas<D>) find_value_kernel(QueryParams p) {
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    const LineView view{p.file, p.n, p.string_index, p.leveled, p.level_size, p.hi, p.marks, p.odd};
    const int64_t per_line = 2 * static_cast<int64_t>(p.slots);
    // lines [first, first + lines); the file's last line ends at p.n
    int64_t first = 0, lines = p.num_lines, file_lines = p.num_lines;
    if (p.range) {
        first = p.range[0];
        lines = p.range[1] - first;
        file_lines = p.last ? p.range[1] : INT64_MAX;
    }
    const int64_t items = query_items(lines, p.num_queries);
    for (int64_t g = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; g < items; g += stride) {
        int64_t li;
        int q;
        if (!query_item(g, 0, lines, p.num_queries, stride, &li, &q)) continue;
        const int64_t i = first + li;
        const bool to_eof = i + 1 >= file_lines;
        if (p.range && (i >= p.out_lines || i + (to_eof ? 0 : 1) >= p.newline_cap)) continue;
        const int64_t start = p.newlines[i];
        const int64_t end = to_eof ? p.n : p.newlines[i + 1];
        if (p.long_lines.items && end - start > p.long_lines.bytes && hand_over(p.long_lines, i, 0, q)) continue;
        int64_t* res = p.out + (static_cast<int64_t>(q) * p.out_lines + i) * per_line;
        const ProgramCode ir{p.programs + p.offsets[q]};
        // writes every slot once, unless a whitespace skip runs far past the
        // line (then a warp evaluates it again)
        int r = run_line<D, SeqScanOf<K>>(view, start, end, ir, res, per_line, kRelLimit,
                                          p.long_lines.items ? p.long_lines.bytes : -1);
        if (r == kLineLong && !hand_over(p.long_lines, i, 0, q)) r = run_line_wide(view, start, end, ir, res, per_line);
        if (r == kLineDeferred) atomicOr(p.status + 1, kErrDeferred);
    }
}

// A warp per item: the lines find_value_kernel handed over, and (by_warp)
// every line of the file, a line's queries side by side.
template <int D>
__global__ void __launch_bounds__(kWarpThreads, kWarpMinCtas<D>) find_value_warp_kernel(QueryParams p) {
    const int64_t warps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
    const int64_t own = p.by_warp ? p.num_lines * p.num_queries : 0;
    const int64_t count = own + handed_over(p.long_lines);
    const LineView view{p.file, p.n, p.string_index, p.leveled, p.level_size, p.hi, p.marks, p.odd};
    const int64_t per_line = 2 * static_cast<int64_t>(p.slots);
    const int64_t file_lines = p.range ? (p.last ? p.range[1] : INT64_MAX) : p.num_lines;
    for (int64_t k = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; k < count; k += warps) {
        LongItem it;
        if (k < own)
            it = LongItem{k / p.num_queries, 0, static_cast<int32_t>(k % p.num_queries)};
        else
            it = p.long_lines.items[k - own];
        const int64_t start = p.newlines[it.line];
        const int64_t end = it.line + 1 >= file_lines ? p.n : p.newlines[it.line + 1];
        int64_t* res = p.out + (static_cast<int64_t>(it.query) * p.out_lines + it.line) * per_line;
        if (run_line<D, WarpScan>(view, start, end, ProgramCode{p.programs + p.offsets[it.query]}, res, per_line) ==
                kLineDeferred &&
            (threadIdx.x & 31) == 0)
            atomicOr(p.status + 1, kErrDeferred);
    }
}

template <int D>
__global__ void __launch_bounds__(kQueryThreads, kQueryMinCtas<D>) find_value_batch_kernel(const QueryFile* files, int nfiles,
                                                                int64_t total_items, LongLines long_lines) {
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t g = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; g < total_items; g += stride) {
        int lo = 0, hi = nfiles - 1;  // last file with item_begin <= g
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (files[mid].item_begin <= g)
                lo = mid;
            else
                hi = mid - 1;
        }
        const QueryFile& F = files[lo];
        int64_t i;
        int q;
        if (!query_item(g - F.item_begin, F.item_begin, F.num_lines, F.num_queries, stride, &i, &q)) continue;
        const LineView view{F.file, F.n, F.string_index, F.leveled, F.level_size, F.n, F.marks, F.odd};
        const int64_t start = F.newlines[i];
        const int64_t end = i + 1 < F.num_lines ? F.newlines[i + 1] : F.n;
        if (long_lines.items && end - start > long_lines.bytes && hand_over(long_lines, i, lo, q)) continue;
        const int64_t per_line = 2 * static_cast<int64_t>(F.slots);
        int64_t* res = F.out + (q * F.out_lines + i) * per_line;
        const ProgramCode ir{F.programs + F.offsets[q]};
        if (run_line<D>(view, start, end, ir, res, per_line, kRelLimit, long_lines.items ? long_lines.bytes : -1) ==
                kLineLong &&
            !hand_over(long_lines, i, lo, q))
            run_line_wide(view, start, end, ir, res, per_line);
    }
}

template <int D>
__global__ void __launch_bounds__(kWarpThreads, kWarpMinCtas<D>) find_value_batch_warp_kernel(const QueryFile* files, int nfiles,
                                                                     int64_t own, LongLines long_lines) {
    const int64_t warps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
    const int64_t count = own + handed_over(long_lines);
    for (int64_t k = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; k < count; k += warps) {
        LongItem it;
        if (k < own) {
            int lo = 0, hi = nfiles - 1;  // last file with warp_begin <= k
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (files[mid].warp_begin <= k)
                    lo = mid;
                else
                    hi = mid - 1;
            }
            const int64_t r = k - files[lo].warp_begin;
            it = LongItem{r / files[lo].num_queries, lo, static_cast<int32_t>(r % files[lo].num_queries)};
        } else {
            it = long_lines.items[k - own];
        }
        const QueryFile& F = files[it.file];
        const LineView view{F.file, F.n, F.string_index, F.leveled, F.level_size, F.n, F.marks, F.odd};
        const int64_t start = F.newlines[it.line];
        const int64_t end = it.line + 1 < F.num_lines ? F.newlines[it.line + 1] : F.n;
        const int64_t per_line = 2 * static_cast<int64_t>(F.slots);
        int64_t* res = F.out + (it.query * F.out_lines + it.line) * per_line;
        run_line<D, WarpScan>(view, start, end, ProgramCode{F.programs + F.offsets[it.query]}, res,
                                    per_line);
    }
}

template <int D>
cudaError_t launch_batch_d(const QueryFile* files, int nfiles, int64_t items, int64_t warp_items,
                           const LongLines& L, int grid, int warp_grid, cudaStream_t stream) {
    cudaError_t e = cudaSuccess;
    if (items > 0) {
        find_value_batch_kernel<D><<<grid, kQueryThreads, 0, stream>>>(files, nfiles, items, L);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess && (L.items || warp_items > 0)) {
        find_value_batch_warp_kernel<D><<<warp_grid, kWarpThreads, 0, stream>>>(files, nfiles, warp_items, L);
        e = cudaGetLastError();
    }
    return e;
}

template <int D>
cudaError_t launch_d(const QueryParams& p, int grid, int warp_grid, cudaStream_t stream) {
    cudaError_t e = cudaSuccess;
    if (!p.by_warp) {
        if (p.short_lines)
            find_value_kernel<D, 1><<<grid, kQueryThreads, 0, stream>>>(p);
        else
            find_value_kernel<D, 2><<<grid, kQueryThreads, 0, stream>>>(p);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess && (p.by_warp || p.long_lines.items)) {
        find_value_warp_kernel<D><<<warp_grid, kWarpThreads, 0, stream>>>(p);
        e = cudaGetLastError();
    }
    return e;
}

}  // namespace

cudaError_t launch_find_value_batch(const QueryFile* files, int nfiles, int64_t items, int64_t warp_items, int depth,
                                    const LongLines& long_lines, int grid, int warp_grid, cudaStream_t stream) {
    switch (level_slots_for_depth(depth)) {
        case 5:
            return launch_batch_d<5>(files, nfiles, items, warp_items, long_lines, grid, warp_grid, stream);
        case 9:
            return launch_batch_d<9>(files, nfiles, items, warp_items, long_lines, grid, warp_grid, stream);
        default:
            return launch_batch_d<kLevelSlots>(files, nfiles, items, warp_items, long_lines, grid, warp_grid, stream);
    }
}

cudaError_t launch_find_value(const QueryParams& p, int grid, int warp_grid, cudaStream_t stream) {
    switch (level_slots_for_depth(p.depth)) {
        case 5:
            return launch_d<5>(p, grid, warp_grid, stream);
        case 9:
            return launch_d<9>(p, grid, warp_grid, stream);
        default:
            return launch_d<kLevelSlots>(p, grid, warp_grid, stream);
    }
}

int find_value_max_ctas_per_sm(int depth) {
    int blocks = 0;
    cudaError_t e;
    switch (level_slots_for_depth(depth)) {
        case 5:
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, find_value_kernel<5, 2>, kQueryThreads, 0);
            break;
        case 9:
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, find_value_kernel<9, 2>, kQueryThreads, 0);
            break;
        default:
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, find_value_kernel<kLevelSlots, 2>, kQueryThreads, 0);
    }
    return e == cudaSuccess ? blocks : -1;
}

}  // namespace gpj
