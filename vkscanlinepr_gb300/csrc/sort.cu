// sort.cu — onesweep LSD radix sort (8-bit digits) for 64- and 32-bit keys
// with 32-bit values.
//
// Replaces naive_seg_sort_pairs.comp:26-97, an O(len^2) odd-even
// transposition sort per path segment.  The fragment key already carries the
// path in its high bits (see pack_key), so one stable sort of the whole
// array by key gives the reference's per-path order by (signed yx, index).
//
// Per pass, each CTA takes tile after tile (from a counter; 8, 12 or 16 keys a
// thread, 3,072 keys by default), ranks keys by
// digit with warp __match_any_sync / popc, publishes its per-digit counts,
// and looks back over earlier tiles' per-digit counts to find where its run
// of each digit starts; the thread of a digit reads the words of 8
// preceding tiles per step, all loads in flight together.  Keys are first
// scattered into shared memory in digit order, then written out in runs, so
// global stores stay mostly contiguous.  An upfront kernel histograms every
// pass's digits in one read of the keys.
#include <algorithm>

#include "kernels.h"
#include "scan.cuh"

namespace sr {

namespace {
constexpr int kRadixBits = 8;
constexpr int kRadix = 1 << kRadixBits;
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
// Keys per thread of a tile: 8, 12 or 16 (chosen per plan; 12 by default).
constexpr uint32_t kFlagA = 1u << 30;
constexpr uint32_t kFlagP = 2u << 30;
constexpr uint32_t kCountMask = (1u << 30) - 1u;
constexpr int kMaxPasses = 8;
constexpr int kHistBlocks = 608;   // 152 SMs x 4
constexpr int kLookWindow = 8;     // look-back words read per step
// Lanes holding the same digit: one __match_any_sync, or one ballot per
// digit bit (9 bits: digit 256 marks an empty slot).  The 64-bit fragment
// keys are ranked by ballots (their low digits vary a lot within a warp);
// the 32-bit keys (draw rows) arrive in runs, where one match is cheaper.
template <bool kMatchAny> SR_DEV uint32_t same_digit_lanes(uint32_t d) {
    if (kMatchAny) return __match_any_sync(0xFFFFFFFFu, d);
    uint32_t peers = 0xFFFFFFFFu;
#pragma unroll
    for (int b = 0; b <= kRadixBits; ++b) {
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, (d >> b) & 1u);
        peers &= ((d >> b) & 1u) ? m : ~m;
    }
    return peers;
}

// Digit of a pass; bits at or above key_bits do not take part.
template <typename K> SR_DEV uint32_t digit_of(K k, uint32_t shift, uint32_t mask) {
    return (uint32_t)(k >> shift) & mask;
}

__host__ __device__ inline uint32_t digit_mask(uint32_t key_bits, uint32_t shift) {
    const uint32_t left = key_bits > shift ? key_bits - shift : 0u;
    return left >= (uint32_t)kRadixBits ? (uint32_t)(kRadix - 1) : ((1u << left) - 1u);
}

struct Scratch {
    uint32_t* hist;       // [passes][256] digit counts
    uint32_t* lookback;   // [passes][tiles + 1][256]
    uint32_t* counters;   // [passes] tile counters
};

Scratch carve(const SortPlan& p, void* base) {
    Scratch s;
    char* b = static_cast<char*>(base);
    s.hist = reinterpret_cast<uint32_t*>(b);
    b += sizeof(uint32_t) * kMaxPasses * kRadix;
    s.counters = reinterpret_cast<uint32_t*>(b);
    b += sizeof(uint32_t) * 64;
    s.lookback = reinterpret_cast<uint32_t*>(b);
    return s;
}
}  // namespace

SortPlan sort_plan(int64_t n, uint32_t key_bits, const uint32_t* n_dev, int items) {
    SortPlan p;
    p.n = n;
    p.n_dev = n_dev;
    p.key_bits = key_bits;
    p.passes = (key_bits + kRadixBits - 1) / kRadixBits;
    if (p.passes == 0) p.passes = 1;
    p.items = items == 8 || items == 16 ? items : 12;
    p.tiles = (uint32_t)((n + kThreads * p.items - 1) / (kThreads * p.items));
    return p;
}

size_t sort_scratch_bytes(const SortPlan& p) {
    return sizeof(uint32_t) * (kMaxPasses * kRadix + 64) +
           sizeof(uint32_t) * (size_t)p.passes * ((size_t)p.tiles + 1) * kRadix;
}

// Histogram of every pass's digits (grid-stride; warp-aggregated shared
// atomics because neighbouring keys usually share their high digits).
template <typename K>
__global__ void __launch_bounds__(kThreads) k_hist(const K* __restrict__ keys, int64_t n_max,
                                                   const uint32_t* __restrict__ n_dev, uint32_t passes,
                                                   uint32_t key_bits, uint32_t* __restrict__ hist) {
    wait_for_stream();
    __shared__ uint32_t sh[kMaxPasses][kRadix];
    const int64_t n = n_dev ? (int64_t)min((uint64_t)*n_dev, (uint64_t)n_max) : n_max;
    for (int i = threadIdx.x; i < kMaxPasses * kRadix; i += kThreads) (&sh[0][0])[i] = 0;
    __syncthreads();
    const uint32_t lane = lane_id();
    int64_t stride = (int64_t)gridDim.x * kThreads;
    for (int64_t i0 = (int64_t)blockIdx.x * kThreads; i0 < n; i0 += stride) {
        int64_t i = i0 + threadIdx.x;
        bool ok = i < n;
        K k = ok ? keys[i] : (K)0;
        uint32_t am = __ballot_sync(0xFFFFFFFFu, ok);
        for (uint32_t p = 0; p < passes; ++p) {
            uint32_t d = digit_of(k, p * kRadixBits, digit_mask(key_bits, p * kRadixBits));
            if (ok) {
                uint32_t peers = __match_any_sync(am, d);
                if (lane == (uint32_t)(__ffs(peers) - 1)) atomicAdd(&sh[p][d], (uint32_t)__popc(peers));
            }
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < passes * kRadix; i += kThreads) {
        uint32_t v = (&sh[0][0])[i];
        if (v) atomicAdd(&hist[i], v);
    }
}

// A tile of rows: their first positions (exclusive scan of the counts), and
// the tile's part of every pass's digit counts (a row is the key of each of
// its records).
constexpr int kRowTile = kThreads * 4;
__global__ void __launch_bounds__(kThreads) k_row_starts(const uint32_t* __restrict__ counts, uint32_t rows,
                                                         int32_t* __restrict__ row_start, uint32_t passes,
                                                         uint32_t key_bits, uint32_t* __restrict__ hist,
                                                         uint64_t* tstat, uint32_t* counter, uint32_t* status,
                                                         uint32_t spin_limit) {
    wait_for_stream();
    __shared__ uint32_t sh[kMaxPasses][kRadix];
    __shared__ uint32_t s_tile;
    __shared__ int32_t s_warp[kWarps + 1];
    if (threadIdx.x == 0) s_tile = atomicAdd(counter, 1u);
    for (uint32_t i = threadIdx.x; i < passes * kRadix; i += kThreads) (&sh[0][0])[i] = 0;
    __syncthreads();
    const uint32_t tile = s_tile;
    // A frame that has failed by now (its caller is told so) has rows without
    // records: where a wait gave up, the counts may add up to more than the
    // order has room for.
    const uint32_t counted = *status ? 0u : rows;
    for (uint32_t q = 0; q < 4; ++q) {
        const uint32_t b = tile * kRowTile + q * kThreads + threadIdx.x;
        const uint32_t c = b < counted ? counts[b] : 0u;
        if (!c) continue;
        for (uint32_t p = 0; p < passes; ++p)
            atomicAdd(&sh[p][digit_of(b, p * kRadixBits, digit_mask(key_bits, p * kRadixBits))], c);
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < passes * kRadix; i += kThreads) {
        const uint32_t v = (&sh[0][0])[i];
        if (v) atomicAdd(&hist[i], v);
    }
    int32_t total;
    int4 v[1];
    load_tile_values<1, kThreads>(v, reinterpret_cast<const int32_t*>(counts), counted, tile);
    scan_tile_values<1, kThreads>(v, row_start, rows, tile, tstat, status, spin_limit, s_warp, &total);
}

// A wait of the row order gave up: some of its places will not be written, and
// the resolve, which would read what they hold, finds the rows empty.
SR_DEV void give_up_rows(int32_t* row_start, uint32_t rows, uint32_t* status) {
    set_error(status, ERR_LOOKBACK_TIMEOUT);
    if (row_start)
        for (uint32_t r = 0; r <= rows; ++r) row_start[r] = 0;
}

// ------------------------------------------------ row sort in one pass ---
// The order of the paint runs by row, stable, for frames of up to 1,024 rows:
// one pass with a digit a row.  The rows' starts are known (k_row_starts), so
// a record's place is its row's start, plus the row's records in earlier tiles
// (a look-back a row, as above: a thread owns every 256th row and looks for all
// of them at once), plus those before it in its tile.  Only the record indices
// are written; they go straight to their places, neighbours in a tile being
// mostly of different rows.  A small frame's row sort is the latency of its
// launches and of the look-back: two launches instead of three took 18 instead
// of 21 us for 1,024 rows and 100,000 runs, 14 instead of 21 for 375 rows (a
// 1000x750 frame of two pixel rows a row).  The look-back words and their
// clearing grow with the rows and the draw records: with 1,024 rows the row
// order of 2.5 M draw records took 30.6 instead of 31.7 us, of 3.3 M 34.7
// instead of 33.7, of 12.4 M 73.6 instead of 62.4; with 400 rows 42.9 instead of
// 54.2 for 10.5 M; with 2,048 rows 57 instead of 40 for a small frame.
constexpr uint32_t kRowSortMaxRows = 1024, kRowSortAnyRows = 512;   // any: whatever the draw records
constexpr int64_t kRowSortMaxDraws = 3500000;
constexpr int kRowItems = 8;
constexpr int kRowWindow = 4;   // look-back words of a row read per step
constexpr int kRowSortTile = kThreads * kRowItems;

template <int BITS>
__global__ void __launch_bounds__(kThreads) k_row_sort(const uint32_t* __restrict__ rows_in, int64_t n_max,
                                                       const uint32_t* __restrict__ n_dev, uint32_t rows,
                                                       int32_t* row_start, uint32_t* __restrict__ idx_out,
                                                       uint32_t* __restrict__ lookback, uint32_t* counter,
                                                       uint32_t* status, uint32_t spin_limit) {
    wait_for_stream();
    constexpr int kR = 1 << BITS, kPer = kR / kThreads;
    __shared__ __align__(16) uint16_t hist[kWarps][kR];
    __shared__ uint32_t base[kR];
    __shared__ uint32_t s_tile;
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    uint4* clear = reinterpret_cast<uint4*>(&hist[0][0]);
    for (int i = threadIdx.x; i < (int)(sizeof(hist) / 16); i += kThreads) clear[i] = make_uint4(0u, 0u, 0u, 0u);
    if (threadIdx.x == 0) s_tile = atomicAdd(counter, 1u);
    __syncthreads();
    const uint32_t tile = s_tile;
    const int64_t n = n_dev ? (int64_t)min((uint64_t)*n_dev, (uint64_t)n_max) : n_max;
    const int64_t tbase = (int64_t)tile * kRowSortTile;
    if (tbase >= n) return;   // launched for a larger capacity than this frame has
    const int64_t wbase = tbase + (int64_t)warp * (32 * kRowItems) + lane;

    // ---- load and rank within the warp
    uint32_t at[kRowItems];   // row << 16 | rank
#pragma unroll
    for (int it = 0; it < kRowItems; ++it)
        at[it] = wbase + it * 32 < n ? rows_in[wbase + it * 32] & (uint32_t)(kR - 1) : (uint32_t)kR;
#pragma unroll
    for (int it = 0; it < kRowItems; ++it) {
        const uint32_t r = at[it];
        const uint32_t peers = __match_any_sync(0xFFFFFFFFu, r);
        const uint32_t leader = (uint32_t)(__ffs(peers) - 1);
        uint32_t before = 0;
        if (r < (uint32_t)kR && lane == leader) {
            before = hist[warp][r];
            hist[warp][r] = (uint16_t)(before + (uint32_t)__popc(peers));
        }
        before = __shfl_sync(0xFFFFFFFFu, before, leader);
        at[it] = (r << 16) | (before + (uint32_t)__popc(peers & lanemask_lt()));
        __syncwarp();
    }
    __syncthreads();

    // ---- per row: offsets across warps, the tile's count published
    uint32_t cnt[kPer];
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
        const uint32_t d = threadIdx.x + (uint32_t)q * kThreads;
        uint32_t c = 0;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            const uint32_t t = hist[w][d];
            hist[w][d] = (uint16_t)c;
            c += t;
        }
        cnt[q] = c;
        if (d < rows) st_relaxed_u32(lookback + (size_t)tile * kR + d, (tile == 0 ? kFlagP : kFlagA) | c);
    }
    // ---- the rows' records in earlier tiles: all of the thread's rows at
    // once, kRowWindow tiles each
    uint32_t excl[kPer];
    int32_t look[kPer];   // < 0: done
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
        excl[q] = 0;
        look[q] = threadIdx.x + (uint32_t)q * kThreads < rows ? (int32_t)tile - 1 : -1;
    }
    uint32_t spins = 0;
    for (;;) {
        uint32_t w[kPer][kRowWindow];
        bool left = false, moved = false;
#pragma unroll
        for (int q = 0; q < kPer; ++q)
#pragma unroll
            for (int k = 0; k < kRowWindow; ++k)
                w[q][k] = look[q] - k >= 0
                              ? ld_relaxed_u32(lookback + (size_t)(look[q] - k) * kR + threadIdx.x + q * kThreads)
                              : kFlagP;
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            if (look[q] < 0) continue;
            int used = 0;
            bool done = false;
#pragma unroll
            for (int k = 0; k < kRowWindow; ++k) {
                if (done || used < k) continue;   // stopped at an earlier word
                const uint32_t f = w[q][k] & ~kCountMask;
                if (f == 0) continue;             // not published yet: used stays k
                excl[q] += w[q][k] & kCountMask;
                used = k + 1;
                done = f == kFlagP;
            }
            look[q] = done ? -1 : look[q] - used;
            moved = moved || used;
            left = left || look[q] >= 0;
        }
        if (!left) break;
        if (!moved) {
            if (++spins > spin_limit) {
                give_up_rows(row_start, rows, status);
                break;
            }
            __nanosleep(32);
        }
    }
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
        const uint32_t d = threadIdx.x + (uint32_t)q * kThreads;
        if (d >= rows) continue;
        if (tile > 0) st_relaxed_u32(lookback + (size_t)tile * kR + d, kFlagP | (excl[q] + cnt[q]));
        base[d] = (uint32_t)row_start[d] + excl[q];
    }
    __syncthreads();

    // ---- to their places
#pragma unroll
    for (int it = 0; it < kRowItems; ++it) {
        const uint32_t r = at[it] >> 16;
        if (r >= rows) continue;
        const uint32_t o = base[r] + hist[warp][r] + (at[it] & 0xFFFFu);
        if ((int64_t)o < n) idx_out[o] = (uint32_t)(wbase + it * 32);
        else set_error(status, ERR_BAD_INDEX);
    }
}

template <typename K, bool kVals, int ITEMS> struct OnesweepSmem {
    uint32_t warp_hist[kWarps][kRadix];
    uint32_t digit_start[kRadix];   // tile-local exclusive start of each digit
    uint32_t digit_global[kRadix];  // global base minus digit_start
    uint2 scan_tmp[kWarps];
    uint32_t tile;
    K keys[kThreads * ITEMS];
    uint32_t vals[kVals ? kThreads * ITEMS : 1];
};

// Resident CTAs per SM the register budget is set for.
constexpr int onesweep_min_blocks(bool vals, int items) {
    return vals ? (items <= 8 ? 4 : items <= 12 ? 3 : 2) : (items <= 8 ? 5 : items <= 12 ? 4 : 3);
}

template <typename K, bool kVals, int ITEMS>
__global__ void __launch_bounds__(kThreads, onesweep_min_blocks(kVals, ITEMS)) k_onesweep(
                                                       const K* __restrict__ keys_in,
                                                       const uint32_t* __restrict__ vals_in,
                                                       K* __restrict__ keys_out, uint32_t* __restrict__ vals_out,
                                                       int64_t n_max, const uint32_t* __restrict__ n_dev,
                                                       uint32_t shift, uint32_t dmask,
                                                       const uint32_t* __restrict__ digit_count,
                                                       uint32_t* __restrict__ lookback, uint32_t* counter,
                                                       int32_t* row_start, uint32_t rows, uint32_t* status,
                                                       uint32_t spin_limit) {
    wait_for_stream();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int kItems = ITEMS, kTile = kThreads * ITEMS;
    OnesweepSmem<K, kVals, ITEMS>& S = *reinterpret_cast<OnesweepSmem<K, kVals, ITEMS>*>(smem_raw);
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    // (rows whose counts were left out, as some look-back before had given up,
    // leave places unwritten too)
    if (row_start && blockIdx.x == 0 && *status != 0u)
        for (uint32_t r = threadIdx.x; r <= rows; r += kThreads) row_start[r] = 0;
    const int64_t n = n_dev ? (int64_t)min((uint64_t)*n_dev, (uint64_t)n_max) : n_max;
    // tile after tile until the input's end: the grid follows the GPU, not the
    // capacity, of which a frame's runs are a fraction (a CTA a tile of the
    // capacity: 0.103 instead of 0.091 ms for the row sort of the 4096^2 frame,
    // 0.105 instead of 0.079 for 64 uneven scenes)
    for (;; __syncthreads()) {
        for (int i = threadIdx.x; i < kWarps * kRadix; i += kThreads) (&S.warp_hist[0][0])[i] = 0;
        if (threadIdx.x == 0) S.tile = atomicAdd(counter, 1u);
        __syncthreads();
        const uint32_t tile = S.tile;
        const int64_t tbase = (int64_t)tile * kTile;
        if (tbase >= n) return;
        const int64_t wbase = tbase + (int64_t)warp * (32 * kItems);

        // ---- load (warp-striped, coalesced) and rank within the warp
        K k[kItems];
        uint32_t v[kVals ? kItems : 1];
        uint32_t rank[kItems];
#pragma unroll
        for (int it = 0; it < kItems; ++it) {
            int64_t idx = wbase + it * 32 + lane;
            bool ok = idx < n;
            k[it] = ok ? keys_in[idx] : (K)0;
            if (kVals) v[it] = ok ? (vals_in ? vals_in[idx] : (uint32_t)idx) : 0u;
        }
#pragma unroll
        for (int it = 0; it < kItems; ++it) {
            int64_t idx = wbase + it * 32 + lane;
            bool ok = idx < n;
            uint32_t d = ok ? digit_of(k[it], shift, dmask) : (uint32_t)kRadix;   // kRadix = out of range
            uint32_t peers = same_digit_lanes<sizeof(K) == 4>(d);
            uint32_t leader = (uint32_t)(__ffs(peers) - 1);
            uint32_t before = 0;
            if (ok && lane == leader) {
                before = S.warp_hist[warp][d];
                S.warp_hist[warp][d] = before + (uint32_t)__popc(peers);
            }
            before = __shfl_sync(0xFFFFFFFFu, before, leader);
            rank[it] = before + (uint32_t)__popc(peers & lanemask_lt());
            __syncwarp();
        }
        __syncthreads();

        // ---- per digit: exclusive offsets across warps; tile count; publish
        const uint32_t d = threadIdx.x;   // kThreads == kRadix
        uint32_t cnt = 0;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            uint32_t t = S.warp_hist[w][d];
            S.warp_hist[w][d] = cnt;
            cnt += t;
        }
        uint32_t* lb_mine = lookback + (size_t)tile * kRadix + d;
        st_relaxed_u32(lb_mine, (tile == 0 ? kFlagP : kFlagA) | cnt);

        // tile-local digit starts and the digits' global starts: block exclusive
        // scans over the tile's 256 counts and over the whole input's
        const uint32_t all = digit_count[d];
        uint32_t x = cnt, y = all;
#pragma unroll
        for (int dd = 1; dd < 32; dd <<= 1) {
            const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, x, dd), u = __shfl_up_sync(0xFFFFFFFFu, y, dd);
            if ((int)lane >= dd) {
                x += t;
                y += u;
            }
        }
        if (lane == 31) S.scan_tmp[warp] = make_uint2(x, y);
        __syncthreads();
        uint32_t dstart = x - cnt, gstart = y - all;
        for (uint32_t w = 0; w < warp; ++w) {
            dstart += S.scan_tmp[w].x;
            gstart += S.scan_tmp[w].y;
        }
        S.digit_start[d] = dstart;

        // ---- look-back for this digit: 8 preceding tiles' words per step, all
        // loads in flight together; stop at the first inclusive prefix, wait
        // (bounded) at the first tile that has published nothing yet
        uint32_t excl = 0;
        if (tile > 0) {
            const uint32_t* base = lookback + d;
            int64_t look = (int64_t)tile - 1;
            uint32_t spins = 0;
            for (;;) {
                uint32_t w[kLookWindow];
#pragma unroll
                for (int q = 0; q < kLookWindow; ++q)
                    w[q] = look - q >= 0 ? ld_relaxed_u32(base + (size_t)(look - q) * kRadix) : kFlagP;
                int used = 0;
                bool done = false;
#pragma unroll
                for (int q = 0; q < kLookWindow; ++q) {
                    if (done || used < q) continue;   // stopped at an earlier word
                    const uint32_t f = w[q] & ~kCountMask;
                    if (f == 0) continue;             // not published yet: used stays q
                    excl += w[q] & kCountMask;
                    used = q + 1;
                    done = f == kFlagP;
                }
                if (done) break;
                look -= used;
                if (used == 0) {
                    if (++spins > spin_limit) {
                        give_up_rows(row_start, rows, status);
                        break;
                    }
                    __nanosleep(32);
                }
            }
            st_relaxed_u32(lb_mine, kFlagP | (excl + cnt));
        }
        S.digit_global[d] = gstart + excl - dstart;
        __syncthreads();

        // ---- scatter into shared memory in digit order
#pragma unroll
        for (int it = 0; it < kItems; ++it) {
            int64_t idx = wbase + it * 32 + lane;
            if (idx < n) {
                uint32_t dg = digit_of(k[it], shift, dmask);
                uint32_t pos = S.digit_start[dg] + S.warp_hist[warp][dg] + rank[it];
                S.keys[pos] = k[it];
                if (kVals) S.vals[pos] = v[it];
            }
        }
        __syncthreads();

        // ---- write runs to global memory
        int64_t valid = n - tbase;
        if (valid > kTile) valid = kTile;
        for (int j = threadIdx.x; j < valid; j += kThreads) {
            K kk = S.keys[j];
            uint32_t dg = digit_of(kk, shift, dmask);
            uint32_t o = S.digit_global[dg] + (uint32_t)j;
            if ((int64_t)o < n) {
                keys_out[o] = kk;
                if (kVals) vals_out[o] = S.vals[j];
            } else {
                set_error(status, ERR_BAD_INDEX);
            }
        }
    }
}

template <typename K, bool kVals, int ITEMS>
static void sort_impl(const SortPlan& p, const K* keys_in, const uint32_t* vals_in, K* keys_out, uint32_t* vals_out,
                      K* keys_alt, uint32_t* vals_alt, void* scratch, uint32_t* status, cudaStream_t st) {
    if (p.n <= 0) return;
    Scratch s = carve(p, scratch);
    if (!p.cleared) cudaMemsetAsync(scratch, 0, sort_scratch_bytes(p), st);
    if (!p.hist_given) {
        int hb = (int)((p.n + kThreads - 1) / kThreads);
        if (hb > kHistBlocks) hb = kHistBlocks;
        count_launches(1);
        launch_after(k_hist<K>, hb, kThreads, 0, st, keys_in, p.n, p.n_dev, p.passes, p.key_bits, s.hist);
    }
    const size_t smem = sizeof(OnesweepSmem<K, kVals, ITEMS>);
    static std::atomic<uint32_t> attr_set{0};
    static std::atomic<uint32_t> wave{1};   // CTAs the GPU holds (the same on every device of the build's architecture)
    once_per_device(attr_set, [&] {
        cudaFuncSetAttribute(k_onesweep<K, kVals, ITEMS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        int dev = 0, sms = 0, per = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_onesweep<K, kVals, ITEMS>, kThreads, smem);
        wave.store((uint32_t)std::max(sms, 1) * (uint32_t)std::max(per, 1));
    });
    const unsigned grid = std::min(p.tiles, wave.load());
    const K* ksrc = keys_in;
    const uint32_t* vsrc = vals_in;
    for (uint32_t pass = 0; pass < p.passes; ++pass) {
        bool to_out = ((p.passes - 1 - pass) % 2) == 0;
        K* kdst = to_out ? keys_out : keys_alt;
        uint32_t* vdst = to_out ? vals_out : vals_alt;
        count_launches(1);
        launch_after(k_onesweep<K, kVals, ITEMS>, grid, kThreads, smem, st, ksrc, vsrc, kdst, vdst, p.n, p.n_dev,
                     pass * kRadixBits, digit_mask(p.key_bits, pass * kRadixBits), s.hist + pass * kRadix,
                     s.lookback + (size_t)pass * (p.tiles + 1) * kRadix, s.counters + pass, p.row_start, p.rows, status,
                     spin_limit());
        ksrc = kdst;
        vsrc = vdst;
    }
}

template <typename K>
static void sort_dispatch(const SortPlan& p, const K* keys_in, const uint32_t* vals_in, K* keys_out, uint32_t* vals_out,
                          K* keys_alt, uint32_t* vals_alt, void* scratch, uint32_t* status, cudaStream_t st) {
#define SR_SORT_CASE(ITEMS)                                                                                        \
    if (p.items == ITEMS) {                                                                                        \
        if (vals_out)                                                                                              \
            sort_impl<K, true, ITEMS>(p, keys_in, vals_in, keys_out, vals_out, keys_alt, vals_alt, scratch, status, \
                                      st);                                                                         \
        else                                                                                                       \
            sort_impl<K, false, ITEMS>(p, keys_in, nullptr, keys_out, nullptr, keys_alt, nullptr, scratch, status,  \
                                       st);                                                                        \
        return;                                                                                                    \
    }
    SR_SORT_CASE(8)
    SR_SORT_CASE(16)
    SR_SORT_CASE(12)
#undef SR_SORT_CASE
}

void launch_sort_u64(const SortPlan& p, const uint64_t* keys_in, const uint32_t* vals_in, uint64_t* keys_out,
                     uint32_t* vals_out, uint64_t* keys_alt, uint32_t* vals_alt, void* scratch, uint32_t* status,
                     cudaStream_t st) {
    sort_dispatch<uint64_t>(p, keys_in, vals_in, keys_out, vals_out, keys_alt, vals_alt, scratch, status, st);
}

bool row_sort_one_pass(int64_t n, uint32_t rows) {
    return rows > (uint32_t)kRadix && rows <= (n <= kRowSortMaxDraws ? kRowSortMaxRows : kRowSortAnyRows);
}

static int row_sort_bits(uint32_t rows) { return rows <= 512 ? 9 : 10; }

size_t row_sort_bytes(int64_t n, uint32_t rows) {
    const size_t tiles = (size_t)((n + kRowSortTile - 1) / kRowSortTile);
    return 256 + sizeof(uint32_t) * (tiles << row_sort_bits(rows));
}

void launch_row_sort(const uint32_t* rows_in, int64_t n, const uint32_t* n_dev, uint32_t rows, int32_t* row_start,
                     uint32_t* idx_out, void* scratch, uint32_t* status, cudaStream_t st) {
    if (n <= 0) return;
    uint32_t* counter = static_cast<uint32_t*>(scratch);
    uint32_t* lookback = counter + 64;
    const unsigned tiles = (unsigned)((n + kRowSortTile - 1) / kRowSortTile);
    count_launches(1);
    const int bits = row_sort_bits(rows);
    if (bits == 9)
        launch_after(k_row_sort<9>, tiles, kThreads, 0, st, rows_in, n, n_dev, rows, row_start, idx_out, lookback,
                     counter, status, spin_limit());
    else
        launch_after(k_row_sort<10>, tiles, kThreads, 0, st, rows_in, n, n_dev, rows, row_start, idx_out, lookback,
                     counter, status, spin_limit());
}

size_t row_scan_words(uint32_t rows) { return (size_t)(rows + kRowTile - 1) / kRowTile + 1; }

void launch_row_starts(SortPlan& p, const uint32_t* row_count, uint32_t rows, int32_t* row_start, void* scratch,
                       uint64_t* tile_status, uint32_t* tile_counter, uint32_t* status, cudaStream_t st) {
    p.cleared = 1;
    p.hist_given = 1;
    p.row_start = row_start;
    p.rows = rows;
    if (rows == 0) {
        cudaMemsetAsync(row_start, 0, sizeof(int32_t), st);
        return;
    }
    count_launches(1);
    launch_after(k_row_starts, (rows + kRowTile - 1) / kRowTile, kThreads, 0, st, row_count, rows, row_start, p.passes,
                 p.key_bits, carve(p, scratch).hist, tile_status, tile_counter, status, spin_limit());
}

void launch_sort_u32(const SortPlan& p, const uint32_t* keys_in, const uint32_t* vals_in, uint32_t* keys_out,
                     uint32_t* vals_out, uint32_t* keys_alt, uint32_t* vals_alt, void* scratch, uint32_t* status,
                     cudaStream_t st) {
    sort_dispatch<uint32_t>(p, keys_in, vals_in, keys_out, vals_out, keys_alt, vals_alt, scratch, status, st);
}

}  // namespace sr
