// Standalone structural index for NDJSON on sm_100a: index builds without
// in-kernel queries (the default), single files and batches of files.
//
// A 16 KiB tile is indexed from its own bytes.  In newline-delimited JSON
// the scan state (Sequential.java:36-128: inside-string flag, level counter)
// at every '\n' is (outside, -1).  So the first '\n' of a tile gives the
// state at the tile's first byte backwards: the string state is the parity of
// the quotes before that '\n', the level is -1 less the level change of the
// brackets before it.  No tile reads another's bytes (but for the
// backslashes just before it) or waits for another, and every word is
// computed once, by the tile that holds it.
//
// A tile without a '\n' (a line longer than a tile) takes its state from the
// tiles before it by a decoupled look-back over the line: every tile
// publishes either its end state or, when it has no '\n' and does not know
// its start, its effect on a state (quote parity, level change when entered
// outside or inside a string).  Tiles are claimed in order from a device
// counter, a tile's claim comes after its CTA's previous tile knows its
// state, and a tile waits only for tiles claimed before it, so the waits end.
//
// The assumption is checked, not trusted: every '\n' of a tile must be
// outside strings at level -1, and the state a tile started from must be the
// one the tile before it ended in (newline_scatter_kernel compares them).
// By induction from the file's first byte the index is then the sequential
// definition's; otherwise the input is flagged and the host rebuilds it with
// the exact carry-propagating kernel (index_exact.cu).
//
// One 64-byte word per thread, its masks in registers from the
// classification to the stores.  Two barriers per tile: after the words'
// quote parities (the string states follow from ballots and eight warp
// summaries), and after their level changes (one shuffle scan).  The level
// split is bit-parallel (split_half), so no lane waits for a denser word.
//
// Bound by integer operations: the ALU pipe is 84 % busy at 256 MiB of tweets
// (128 us, DRAM bytes = input + index, 0.40 warp instructions per byte),
// DRAM at 43 % of its rate.  The kernel this one replaced (30 KiB tiles
// with a 2 KiB look-ahead each, word state kept in shared memory between two
// passes, the level split dealt over the warp by cuts) took 193 us there.
// Index builds: 2 GiB of tweets 1558 -> 1076 us; 1 GiB with lines up to 1 MiB,
// which went to the exact kernel before, 1287 -> 833 us; 256 MiB of it at 16
// levels 900 -> 263 us; 256 MiB of 117-byte lines 269 -> 166 us.
#include <cstdint>

#include "device_common.cuh"
#include "index_kernel.h"
#include "tile_common.cuh"
#include "word_ops.cuh"

namespace gpj {

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int64_t kTile = kStandaloneTileBytes;
static_assert(kTile == 64 * kThreads, "one word per thread");
constexpr int kFar = 1 << 20;  // a level no tile can reach a marked level from
constexpr int kBefore = 16;  // bytes before the tile kept with it (escapes)

// Tile states, three words per tile (tagged with the launch epoch in the top
// 16 bits where other tiles poll them):
//   [0] effect of a tile without '\n': e(1) | q(1) | dd0 + 16384 (16) | ddt + 16384 (16);
//       e: of a tile of backslashes alone, the escape state of its first byte
//   [1] end state: s(1) | d + 2^46 (47)
//   [2] start state, as [1] (read after the launch only)
constexpr unsigned long long kPayload = (1ull << 48) - 1;

__device__ __forceinline__ unsigned long long tagged(uint32_t epoch, unsigned long long payload) {
    return (static_cast<unsigned long long>(epoch) << 48) | (payload & kPayload);
}
__device__ __forceinline__ bool has_tag(unsigned long long w, uint32_t epoch) {
    return static_cast<uint32_t>(w >> 48) == epoch;
}
__device__ __forceinline__ unsigned long long pack_state(int s, int64_t d) {
    return (static_cast<unsigned long long>(s & 1) << 47) | static_cast<unsigned long long>(d + (1ll << 46));
}
// A state word stands alone, so relaxed accesses suffice.
__device__ __forceinline__ void st_state(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long ld_state(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

struct __align__(128) Shared {
    // TMA destination: up to kBefore bytes before the tile (not for a file's
    // first tile), then the tile at slot + 128
    uint8_t slot[128 + kTile];
    uint64_t full;            // its barrier (phase k & 1 for the CTA's k-th tile)
    TileFile desc[2];         // the file of the k-th tile in [k & 1]
    int64_t tile[2];          // its number
    // per warp: bit 0 quote parity, bit 1 a '\n', bit 2 quote parity before its first '\n'
    uint8_t parity[2][kWarps];
    // per warp: level change (low 16 bits, signed) + newlines << 16
    int32_t change[2][kWarps];
    int32_t first[2];  // level change from the start of the first '\n''s warp up to it
    alignas(8) uint8_t passes[kWarps];  // the warp's words are backslashes alone
    // the look-back's sums and result
    int32_t dd0[kWarps], ddt[kWarps];
    int32_t s0;
    int64_t d0;
    // the launch's, for escape_before (arguments cost the kernel registers)
    const unsigned long long* states;
    unsigned long long* status;
    uint32_t epoch;
    uint32_t escape;  // escape state of the tile's first byte, where a backslash is before it
};

__device__ __forceinline__ uint8_t* tile_bytes(Shared& sh) { return sh.slot + 128; }

// Claims the next tile and starts its copy (one thread).  The tile's number
// and file are in place before the copy's arrive, so the threads that wait
// for the copy see them.  Its 16 bytes of the tile before come along.
__device__ __forceinline__ void claim_tile(const IndexParams& p, Shared& sh, uint32_t k) {
    const int64_t t = p.tile_begin + static_cast<int64_t>(atomicAdd(p.tile_counter, 1u));
    sh.tile[k & 1] = t;
    if (t >= p.tile_end) {
        mbar_arrive(&sh.full);
        return;
    }
    TileFile& F = sh.desc[k & 1];
    fetch_tile_file(p, t, &F);
    const int64_t start = (t - F.tile_begin) * kTile;
    const int64_t bytes = F.n - start < kTile ? F.n - start : kTile;
    const int lead = start > 0 ? kBefore : 0;
    load_slot(F.file, start - lead, bytes + lead, tile_bytes(sh) - lead, &sh.full);
}

// Parity of the run of backslashes that ends the 16 bytes of v, -1 where they
// are all backslashes.
__device__ __forceinline__ int run_at_end(const uint4& v) {
    const uint32_t w = ~eq_bytes(v.w, 0x5C5C5C5Cu) & 0x80808080u, z = ~eq_bytes(v.z, 0x5C5C5C5Cu) & 0x80808080u;
    const uint32_t y = ~eq_bytes(v.y, 0x5C5C5C5Cu) & 0x80808080u, x = ~eq_bytes(v.x, 0x5C5C5C5Cu) & 0x80808080u;
    const uint32_t d = w ? w : (z ? z : (y ? y : x));  // four more bytes do not change the parity
    return d ? (clz32(d) >> 3) & 1 : -1;
}

// The answer of the first lane that has one, or -1.
__device__ __forceinline__ int first_answer(int mine) {
    const unsigned has = __ballot_sync(~0u, mine >= 0);
    return has ? __shfl_sync(~0u, mine, __ffs(static_cast<int>(has)) - 1) : -1;
}

// Escape state of the byte at `w` (a multiple of 16) bytes into the tile of
// buffer b: parity of the run of backslashes before it.  A whole warp calls
// it, where the byte before is a backslash: 16 bytes a lane, back through the
// slot and then the tile before in device memory (four loads in flight).  A
// tile before that is backslashes throughout passes on the state of its own
// first byte, which it publishes with its effect, so a run of any length costs
// each of its tiles one such look and one wait: bound by that chain, 1.4 us a
// tile (a build with one run of 33 MiB 3.0 ms, of 512 MiB 47 ms; of as many
// other bytes 0.07 and 0.5 ms).  Each word for itself walking back to the
// run's first byte costs the square of its length.
__device__ __forceinline__ uint32_t parity_before(Shared& sh, int b, int w) {
    const int lane = threadIdx.x & 31;
    const uint8_t* const bytes = tile_bytes(sh);
    const int64_t tile_start = (sh.tile[b] - sh.desc[b].tile_begin) * kTile;
    const int floor = tile_start > 0 ? -kBefore : 0;
    for (int at = w; at > floor; at -= 512) {
        const int a = at - 16 * (lane + 1);
        const int r = first_answer(a >= floor ? run_at_end(*reinterpret_cast<const uint4*>(bytes + a))
                                              : (tile_start > 0 ? -1 : 0));
        if (r >= 0) return static_cast<uint32_t>(r);
    }
    if (tile_start == 0) return 0;
    const uint8_t* const tile_before = sh.desc[b].file + (tile_start - kTile);
    for (int at = static_cast<int>(kTile) - kBefore; at > 0; at -= 4 * 512) {
        int mine[4];
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const int a = at - 512 * c - 16 * (lane + 1);
            mine[c] = a >= 0 ? run_at_end(*reinterpret_cast<const uint4*>(tile_before + a)) : -1;
        }
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const int r = first_answer(mine[c]);
            if (r >= 0) return static_cast<uint32_t>(r);
        }
    }
    if (tile_start == kTile) return 0;  // the run begins with the file
    const unsigned long long* const before = sh.states + 3 * (sh.tile[b] - 1);
    for (unsigned polls = 1;; ++polls) {
        const unsigned long long g = __shfl_sync(~0u, ld_state(before), 0);
        if (has_tag(g, sh.epoch)) return static_cast<uint32_t>((g >> 33) & 1);
        const bool expired =
            polls > kMaxPolls || ((polls & 1023u) == 0 && __any_sync(~0u, (ld_acquire(sh.status + 1) & kFatalErrors) != 0));
        if (expired) {
            if (lane == 0) atomicOr(sh.status + 1, kErrLookbackTimeout);
            return 0;  // the host reports the error; outputs are not valid
        }
        __nanosleep(64);
    }
}

// The same, out of line (inline it costs the kernel registers); the tile's first
// byte's is kept for the tile after it.
__device__ __noinline__ uint32_t escape_before(Shared& sh, int b, int w) {
    const uint32_t e = parity_before(sh, b, w);
    if (threadIdx.x == 0) sh.escape = e;
    return e;
}

// State before tile t of a file whose first tile is t0 (one warp): the tiles
// before it, back to one whose end state is known.
__device__ void look_back(const unsigned long long* states, int64_t t, int64_t t0, uint32_t epoch,
                          unsigned long long* status, int* s_out, int64_t* d_out) {
    const int lane = threadIdx.x & 31;
    int q = 0;  // effect of the tiles passed, up to tile t
    int64_t dd0 = 0, ddt = 0;
    int64_t base = t - 1;
    int s = 0;
    int64_t d = -1;
    unsigned polls = 0;
    for (;;) {
        const int64_t i = base - lane;
        int kind = 2;  // 0 not ready, 1 effect, 2 state
        int mq = 0, ms = 0;
        int64_t m0 = 0, mt = 0, md = -1;
        if (i >= t0) {
            const unsigned long long e = ld_state(states + 3 * i + 1);
            if (has_tag(e, epoch)) {
                ms = static_cast<int>((e >> 47) & 1);
                md = static_cast<int64_t>(e & ((1ull << 47) - 1)) - (1ll << 46);
            } else {
                const unsigned long long g = ld_state(states + 3 * i);
                kind = has_tag(g, epoch) ? 1 : 0;
                mq = static_cast<int>((g >> 32) & 1);
                m0 = static_cast<int>((g >> 16) & 0xFFFF) - 16384;
                mt = static_cast<int>(g & 0xFFFF) - 16384;
            }
        }
        const unsigned known = __ballot_sync(~0u, kind == 2);
        const unsigned missing = __ballot_sync(~0u, kind == 0);
        const int first = known ? __ffs(known) - 1 : 32;
        const unsigned need = first == 32 ? ~0u : ((1u << first) - 1);
        if (missing & need) {
            ++polls;
            const bool expired =
                polls > kMaxPolls || ((polls & 1023u) == 0 && (ld_acquire(status + 1) & kFatalErrors) != 0);
            if (expired) {
                if (lane == 0) atomicOr(status + 1, kErrLookbackTimeout);
                break;  // the host reports the error; outputs are not valid
            }
            __nanosleep(64);
            continue;
        }
        if (lane >= first) {
            mq = 0;
            m0 = mt = 0;
        }
        // compose the window: higher lanes are earlier tiles
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int eq = __shfl_down_sync(~0u, mq, off);
            const int64_t e0 = __shfl_down_sync(~0u, m0, off), et = __shfl_down_sync(~0u, mt, off);
            if (lane + off < 32) {
                m0 = e0 + (eq ? mt - m0 : m0);
                mt += et;
                mq ^= eq;
            }
        }
        const int wq = __shfl_sync(~0u, mq, 0);
        const int64_t w0 = __shfl_sync(~0u, m0, 0), wt = __shfl_sync(~0u, mt, 0);
        dd0 = w0 + (wq ? ddt - dd0 : dd0);
        ddt += wt;
        q ^= wq;
        if (first < 32) {
            const int fs = __shfl_sync(~0u, ms, first);
            const int64_t fd = __shfl_sync(~0u, md, first);
            s = fs ^ q;
            d = fd + (fs ? ddt - dd0 : dd0);
            break;
        }
        base -= 32;
    }
    *s_out = s;
    *d_out = d;
}

// Registers set the CTAs per SM (one 16 KiB slot each): 40 a thread for up to
// eight levels, 48 with 16, at the price of a few spilled bytes (5, 4 and 3
// CTAs, none spilled: 2 GiB of tweets 1114 us instead of 1102, 1 GiB with
// lines up to 1 MiB at 5 levels 980 instead of 888, 256 MiB of it at 16 levels
// 302 instead of 276).
template <int LV>
__global__ void __launch_bounds__(kThreads, LV <= 8 ? 6 : 5) tile_index_kernel(IndexParams p) {
    __shared__ Shared sh;
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(~0u, tid >> 5, 0);
    const unsigned lt_mask = (1u << lane) - 1;
    uint8_t* const bytes = tile_bytes(sh);
    if (tid == 0) {
        sh.states = p.tile_state;
        sh.status = p.status;
        sh.epoch = p.epoch;
        mbar_init(&sh.full, 1);
        fence_mbar_init();
        claim_tile(p, sh, 0);
    }
    __syncthreads();
    for (uint32_t k = 0;; ++k) {
        const int b = k & 1;
        if (!mbar_wait_bounded(&sh.full, k & 1) && tid == 0) atomicOr(p.status + 1, kErrCopyTimeout);
        const int64_t t = sh.tile[b];
        if (t >= p.tile_end) break;
        const TileFile& F = sh.desc[b];
        const int64_t tile_start = (t - F.tile_begin) * kTile;
        const bool tail = F.n - tile_start < kTile;  // the file ends inside the tile

        // ---- classify the thread's 64 bytes; odd pairs of threads read the
        // 16-byte halves of each 32 bytes in the other order (4 of 8 bank
        // groups per quarter-warp instead of 2)
        uint64_t open, close, structural, colon, newline, p0;
        unsigned ballot_b;  // the warp's words with backslashes
        {
            const bool swapped = (lane & 2) != 0;
            const uint4* even = reinterpret_cast<const uint4*>(bytes + 64 * tid + (swapped ? 16 : 0));
            const uint4* odd = reinterpret_cast<const uint4*>(bytes + 64 * tid + (swapped ? 0 : 16));
            uint32_t v[16];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint4 q = (i & 1 ? odd : even)[i & 2];
                v[4 * i] = q.x, v[4 * i + 1] = q.y, v[4 * i + 2] = q.z, v[4 * i + 3] = q.w;
            }
            uint32_t b0, q0, n0, o0, c0, s0, k0, b1, q1, n1, o1, c1, s1, k1;
            classify32(v, b0, q0, n0, o0, c0, s0, k0, swapped);
            classify32(v + 8, b1, q1, n1, o1, c1, s1, k1, swapped);
            uint64_t bs = (static_cast<uint64_t>(b1) << 32) | b0;
            uint64_t quote = (static_cast<uint64_t>(q1) << 32) | q0;
            newline = (static_cast<uint64_t>(n1) << 32) | n0;
            open = (static_cast<uint64_t>(o1) << 32) | o0;
            close = (static_cast<uint64_t>(c1) << 32) | c0;
            structural = (static_cast<uint64_t>(s1) << 32) | s0;
            colon = (static_cast<uint64_t>(k1) << 32) | k0;
            if (tail) {
                const uint64_t valid = bits_between(0, F.n - tile_start - 64 * tid);
                bs &= valid, quote &= valid, newline &= valid, open &= valid, close &= valid;
                structural &= valid, colon &= valid;
            }
            // escapes: a word's first byte from the run that ends the word
            // before it; a warp without backslashes can only have its first
            // byte escaped
            ballot_b = __ballot_sync(~0u, bs != 0);
            const int first = 64 * 32 * warp;
            uint32_t cin = 0;  // of the warp's first byte
            if ((warp > 0 || tile_start > 0) && bytes[first - 1] == '\\') cin = escape_before(sh, b, first);
            if (ballot_b) {
                // (a word of backslashes passes on what it was given)
                const unsigned runs = __ballot_sync(~0u, trailing_run_odd(bs));
                const unsigned stops = ~__ballot_sync(~0u, bs == ~0ull) & lt_mask;
                if (stops) cin = (runs >> (31 - clz32(stops))) & 1u;
                quote &= ~escaped_bytes(bs, cin);
            } else {
                quote &= ~static_cast<uint64_t>(lane ? 0u : cin);
            }
            p0 = prefix_xor_halves(quote);
        }
        // ---- string states: quote parities by ballot, one byte per warp
        const unsigned ballot_q = __ballot_sync(~0u, static_cast<int>(p0 >> 63) != 0);
        const unsigned ballot_n = __ballot_sync(~0u, newline != 0);
        const int s_lane = __popc(ballot_q & lt_mask) & 1;
        const int nl_lane = ballot_n ? __ffs(ballot_n) - 1 : 0;  // the lane of the warp's first '\n'
        const int nl_bit = newline ? ctz64(newline) : 0;
        if (lane == nl_lane)
            sh.parity[b][warp] = static_cast<uint8_t>(
                (__popc(ballot_q) & 1) | (ballot_n ? 2 : 0) | ((s_lane ^ (static_cast<int>(p0 >> nl_bit) & 1)) << 2));
        __syncthreads();  // the tile's bytes are read
        const uint64_t warps = *reinterpret_cast<const uint64_t*>(sh.parity[b]);
        const uint64_t warps_q = warps & 0x0101010101010101ull, warps_n = warps & 0x0202020202020202ull;
        const int s_warp = (popc64(warps_q & ((1ull << (8 * warp)) - 1)) & 1) ^ s_lane;
        const int nl_warp = warps_n ? ctz64(warps_n) >> 3 : 0;  // the warp of the tile's first '\n'
        const bool first_tile = tile_start == 0;
        int s0 = 0;        // the state before the tile
        int d0 = -1;       // (clamped: a tile moves the level by at most 16384)
        const bool looked_back = !first_tile && !warps_n;
        if (!first_tile) {
            if (warps_n) {
                s0 = (popc64(warps_q & ((1ull << (8 * nl_warp)) - 1)) & 1) ^ (static_cast<int>(warps >> (8 * nl_warp + 2)) & 1);
            } else {
                // no '\n': publish the tile's effect, look back for its start
                const uint64_t outside = ~(p0 ^ (s_warp ? ~0ull : 0ull));
                const int dd0 = __reduce_add_sync(~0u, popc64(open & outside) - popc64(close & outside));
                const int ddt = __reduce_add_sync(~0u, popc64(open) - popc64(close));
                // a tile of backslashes alone (its words still lie in the slot)
                bool passes = ballot_b == ~0u && !tail;
                if (passes) {
#pragma unroll
                    for (int i = 0; i < 4; i++)
                        passes = passes && run_at_end(*reinterpret_cast<const uint4*>(bytes + 64 * tid + 16 * i)) < 0;
                    passes = __all_sync(~0u, passes);
                }
                if (lane == 0) {
                    sh.dd0[warp] = dd0;
                    sh.ddt[warp] = ddt;
                    sh.passes[warp] = passes ? 1 : 0;
                }
                __syncthreads();
                if (warp == 0) {
                    if (lane == 0) {
                        const bool all_pass = *reinterpret_cast<const uint64_t*>(sh.passes) == 0x0101010101010101ull;
                        const unsigned long long escape = all_pass && bytes[-1] == '\\' ? sh.escape : 0;
                        int e0 = 0, et = 0;
#pragma unroll
                        for (int w = 0; w < kWarps; w++) {
                            e0 += sh.dd0[w];
                            et += sh.ddt[w];
                        }
                        st_state(p.tile_state + 3 * t,
                                 tagged(p.epoch, (escape << 33) |
                                                     (static_cast<unsigned long long>(popc64(warps_q) & 1) << 32) |
                                                     (static_cast<unsigned long long>(e0 + 16384) << 16) |
                                                     static_cast<unsigned long long>(et + 16384)));
                    }
                    int s;
                    int64_t d;
                    look_back(p.tile_state, t, F.tile_begin, p.epoch, p.status, &s, &d);
                    if (lane == 0) {
                        sh.s0 = s;
                        sh.d0 = d;
                    }
                }
                __syncthreads();
                s0 = sh.s0;
                d0 = static_cast<int>(sh.d0 > kFar ? kFar : (sh.d0 < -kFar ? -kFar : sh.d0));
            }
        }
        // ---- the masks outside strings; levels by a scan of their changes
        const uint64_t in_string = p0 ^ ((s0 ^ s_warp) ? ~0ull : 0ull);
        open &= ~in_string;
        close &= ~in_string;
        structural &= ~in_string;
        colon &= ~in_string;
        // for find_value's key searches: the marks are the ':' and the quotes
        // that open a string; a word is odd that has a backslash or a ':'
        // not right after a closing quote (or not known to be: the first
        // byte of a warp's words)
        const uint64_t state_before = (in_string << 1) | static_cast<uint64_t>(s0 ^ s_warp);
        const uint64_t closing = ~in_string & state_before;
        const unsigned last_closes = __ballot_sync(~0u, static_cast<int>(closing >> 63) != 0);
        const uint64_t after_closing = (closing << 1) | ((lane ? last_closes >> (lane - 1) : 0u) & 1u);
        const unsigned odd = ballot_b | __ballot_sync(~0u, (colon & ~after_closing) != 0);
        const uint64_t marks = colon | (in_string & ~state_before);
        const uint32_t open_lo = static_cast<uint32_t>(open), open_hi = static_cast<uint32_t>(open >> 32);
        const uint32_t close_lo = static_cast<uint32_t>(close), close_hi = static_cast<uint32_t>(close >> 32);
        const int o_lo = popc32(open_lo), c_lo = popc32(close_lo);
        const int opens = o_lo + popc32(open_hi), closes = c_lo + popc32(close_hi);
        const int change = opens - closes;
        int incl = change + (popc64(newline) << 16);
        const int mine = incl;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int o = __shfl_up_sync(~0u, incl, off);
            if (lane >= off) incl += o;
        }
        if (lane == 31) sh.change[b][warp] = incl;
        const int d_lane = static_cast<int16_t>((incl - mine) & 0xFFFF);
        if (warp == nl_warp && lane == nl_lane && ballot_n) {
            const uint64_t below = (1ull << nl_bit) - 1;
            sh.first[b] = d_lane + popc64(open & below) - popc64(close & below);
        }
        __syncthreads();
        const int warp_change = lane < kWarps ? sh.change[b][lane] : 0;
        int warp_incl = warp_change;
#pragma unroll
        for (int off = 1; off < kWarps; off <<= 1) {
            const int o = __shfl_up_sync(~0u, warp_incl, off);
            if (lane >= off) warp_incl += o;
        }
        const int warp_excl = warp_incl - warp_change;
        const int d_warp = static_cast<int16_t>(__shfl_sync(~0u, warp_excl, warp) & 0xFFFF);
        const int total = __shfl_sync(~0u, warp_incl, kWarps - 1);
        if (!first_tile && warps_n)
            d0 = -1 - static_cast<int16_t>(__shfl_sync(~0u, warp_excl, nl_warp) & 0xFFFF) - sh.first[b];
        if (tid == 0) {
            const int d_total = static_cast<int16_t>(total & 0xFFFF);
            const int64_t d_start = looked_back ? sh.d0 : d0;
            st_state(p.tile_state + 3 * t + 1,
                     tagged(p.epoch, pack_state(s0 ^ (popc64(warps_q) & 1), d_start + d_total)));
            p.tile_state[3 * t + 2] = pack_state(s0, d_start);
            p.tile_newlines[t] = static_cast<int32_t>(static_cast<uint32_t>(total - d_total) >> 16);
            claim_tile(p, sh, k + 1);
        }
        // ---- level split
        const int depth = d0 + d_warp + d_lane, depth_hi = depth + o_lo - c_lo;
        uint64_t lv[LV];
        uint64_t base_level;  // the bytes at level -1
        if (split_range_ok<LV>(depth, o_lo, c_lo) && split_range_ok<LV>(depth_hi, opens - o_lo, closes - c_lo)) {
            uint32_t lo[LV], hi[LV], m_lo, m_hi;
            split_half<LV>(open_lo, close_lo, static_cast<uint32_t>(structural), depth, lo, m_lo);
            split_half<LV>(open_hi, close_hi, static_cast<uint32_t>(structural >> 32), depth_hi, hi, m_hi);
#pragma unroll
            for (int l = 0; l < LV; l++) lv[l] = (static_cast<uint64_t>(hi[l]) << 32) | lo[l];
            base_level = (static_cast<uint64_t>(m_hi) << 32) | m_lo;
        } else if (split_above<LV>(depth, c_lo) && split_above<LV>(depth_hi, closes - c_lo)) {
            // above all levels, no byte at level -1.  Kept out of the first
            // branch's words by a mask instead, this costs every word of
            // tweets 2 % (1 GiB, lines up to 1 MiB: 752 us at 4 levels, 845 at
            // 5; so 709 and 837; by the loop below 770 and 869)
#pragma unroll
            for (int l = 0; l < LV; l++) lv[l] = 0;
            base_level = 0;
        } else {
            split_levels<LV>(open, close, structural, depth, lv);
            base_level = 0;
            for (uint64_t c = newline; c; c &= c - 1) {
                const uint64_t bit = c & (~c + 1), below = bit - 1;
                if (depth + popc64(open & below) - popc64(close & below) == -1) base_level |= bit;
            }
        }
        // every '\n' must be outside strings at level -1
        if (newline & (in_string | ~base_level)) atomicOr(F.status + 1, kErrIrregular);
        // ---- the word to the index
        if (!tail || 64 * tid < F.n - tile_start) {
            const int64_t word = (tile_start >> 6) + tid;
            const uint64_t valid = tail ? bits_between(0, F.n - tile_start - 64 * tid) : ~0ull;
            F.string_index[word] = in_string & valid;
            F.newline_bits[word] = newline;
            if (F.marks) {
                F.marks[word] = marks;
                if (lane == 0) F.odd[word >> 5] = odd;
            }
#pragma unroll
            for (int l = 0; l < LV; l++)
                if (l < p.num_levels) F.leveled[F.level_size * l + word] = lv[l];
        }
    }
}

template <int LV>
int occupancy() {
    int blocks = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, tile_index_kernel<LV>, kThreads, 0) != cudaSuccess)
        return -1;
    return blocks;
}

}  // namespace

int tile_index_max_ctas_per_sm(int lv) {
    if (lv <= 4) return occupancy<4>();
    if (lv <= 8) return occupancy<8>();
    return occupancy<16>();
}

cudaError_t launch_tile_index_kernel(const IndexParams& p, int grid, cudaStream_t stream) {
    if (p.num_levels <= 4)
        tile_index_kernel<4><<<grid, kThreads, 0, stream>>>(p);
    else if (p.num_levels <= 8)
        tile_index_kernel<8><<<grid, kThreads, 0, stream>>>(p);
    else
        tile_index_kernel<16><<<grid, kThreads, 0, stream>>>(p);
    return cudaGetLastError();
}

}  // namespace gpj
