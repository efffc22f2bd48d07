// segsort.cu — the fragment sort, using the order the records arrive in.
//
// Records are written per curve and curves are grouped by path, so the keys
// (path | row rank | x, see pack_key) arrive sorted by path: only the records
// of each path need ordering.  Each path is a segment of the record array.
//   * Segments of at most kGroup records are packed by where they start: the
//     segments starting in [g*kGroup, (g+1)*kGroup) form one tile of at most
//     kTile records, sorted in shared memory by one CTA.
//   * Larger segments are cut into kTile-record chunks, each sorted the same
//     way, then merged pairwise (merge path), as many rounds as the segment
//     needs.
// Both steps are stable, so the result equals a stable sort of the whole
// array by key: the order the onesweep radix sort produces.  Keys may carry a
// payload above the key bits; it moves with its key and takes no part in the
// order.  Work is handed out through a table of tile descriptors built on
// the device, one per CTA, so no CTA searches for its work.
#include <algorithm>

#include "kernels.h"
#include "segtiles.cuh"

namespace sr {

namespace {
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kRadixBits = 9;   // digits of the 64-bit tile sort
constexpr int kRadix = 1 << kRadixBits;

size_t round256(size_t b) { return (b + 255) & ~(size_t)255; }
size_t scan_area(uint32_t P) { return round256(8 * ((size_t)P / kSegThreads + 2)); }

// Tiles of a frame: at most one group tile per kGroup records (a head starts
// its own group; paths without records may make an empty one), plus the
// chunks of large segments (at most one partial chunk per large segment, of
// which there are fewer than cap / kGroup), and never more than the segments
// plus cap / kTile.
size_t max_tiles(uint32_t P, int64_t cap) {
    const size_t per_tile = (size_t)((cap + kTile - 1) / kTile);
    return std::min<size_t>((size_t)P + 2 + per_tile, 5 * per_tile + 2);
}

TileTables carve(const SegArgs& a) {
    TileTables t;
    const size_t mt = max_tiles(a.n_paths, a.cap);
    char* b = static_cast<char*>(a.tables);
    t.desc = reinterpret_cast<uint4*>(b);
    b += round256(mt * 16);
    t.chunks = reinterpret_cast<uint32_t*>(b);
    t.mt = (uint32_t)mt;
    b += round256(kMergeClasses * mt * 4);
    t.fallback = reinterpret_cast<uint32_t*>(b);
    char* z = static_cast<char*>(a.zeroed);
    t.ctl = reinterpret_cast<uint32_t*>(z);
    z += 256;
    t.scan_status = reinterpret_cast<uint64_t*>(z);
    z += scan_area(a.n_paths);
    t.tile_end = reinterpret_cast<uint32_t*>(z);
    t.wide_count = a.wide_count;
    return t;
}

}  // namespace

// -------------------------------------------------------------- tile tables
__global__ void k_seg_largest(const SegArgs s) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= s.n_paths) return;
    uint32_t a, e;
    seg_span(s, p, a, e);
    seg_note_size(s, e - a, nullptr);
}

__global__ void __launch_bounds__(kSegThreads) k_seg_tiles(const SegArgs s, TileTables u, uint32_t* status,
                                                           uint32_t spin_limit) {
    wait_for_stream();
    seg_tiles(s, u, status, spin_limit);
}

// ----------------------------------------------------------- local sort ---
// A tile is sorted by one CTA of a persistent kernel (one wave; tiles come
// from a counter, so the grid does not follow the table's bound on them).
//   * The tile reaches shared memory by one bulk copy (TMA) of its 16-byte
//     aligned span; an odd last key comes by a plain load.
//   * k_tile_sort spreads the records over up to 4096 bins, in key order: the
//     tile's paths in turn, each with bins for its part of the range of (row,
//     x) and one each for its off-canvas records and for row 0 (BinPlan).  A
//     shared atomic gives a record its place in its bin; then a thread counts
//     the records of its slot's bin that come before (by the code below the
//     bin, then by index: the sort is stable) and writes the key to its place.
//     Bins hold some eight records, so the count is short, and a record is
//     moved once instead of once a digit: digit passes (2.3 a record, each a
//     match, two histogram updates and a scatter) took 340 us for the 21 M
//     records of a 4096^2 frame, this takes 276, and 21 instead of 38 us for a
//     stage of 0.37 M records.  It is bound by instructions: the counts a
//     third, the rest spread over the phases.  512 threads and 2 CTAs an SM
//     (256 and 3: 266 us, but 29 for the small frame; 512 and 3, 40 registers:
//     27).  8192 and 16384 bins cost more to clear and scan than they save.
//     Off-canvas records share one key a path, so counting would be quadratic:
//     their place is by index, from ballots.
//   * A tile with a bin of more than 384 records, or with too many paths for
//     the bins, and every tile of a frame that has failed by now, is sorted by
//     digit passes: compact 32-bit items ((path - pmin,
//     row-rank code, x - xmin) in the fewest bits, the payload above), 8-bit
//     digits ranked per warp (match_any and a histogram a warp), scanned and
//     scattered.  (At 128 records 465 instead of 457 us for the stage, at 1024
//     no change.)
//   * A tile whose compact fields and payload do not fit 32 bits is handed to
//     k_local_sort, whose items are 64-bit (rank - rmin codes, the payload in
//     the high word, or the raw key when the fields need more than 32 bits),
//     sorted through global memory by 9-bit digits.

// Fields of a key: path, row rank, x and the payload above them.  Row rank
// and x share the low word (at most 31 bits), so a funnel shift takes the path.
struct KeyFields {
    uint32_t xb, rb, pb;
    uint32_t off_rank;   // rank of the off-canvas records (Hy - 1); row 0 ranks one above
    SR_DEV uint32_t x(uint64_t k) const { return (uint32_t)k & ((1u << xb) - 1u); }
    SR_DEV uint32_t r(uint64_t k) const { return ((uint32_t)k >> xb) & ((1u << rb) - 1u); }
    SR_DEV uint32_t p(uint64_t k) const {
        return __funnelshift_r((uint32_t)k, (uint32_t)(k >> 32), xb + rb) & ((1u << pb) - 1u);
    }
    SR_DEV uint32_t pay(uint64_t k) const {
        return kbits() >= 32u ? (uint32_t)(k >> 32) >> (kbits() - 32u)
                              : __funnelshift_r((uint32_t)k, (uint32_t)(k >> 32), kbits());
    }
    SR_DEV uint32_t kbits() const { return xb + rb + pb; }
};

SR_DEV uint32_t bits_of(uint32_t v) { return v ? 32u - (uint32_t)__clz((int)v) : 0u; }
SR_DEV uint32_t low_mask(uint32_t b) { return b >= 32 ? 0xFFFFFFFFu : (1u << b) - 1u; }

// Shared memory of the pass machinery and the range reduction.
struct PassSmem {
    uint32_t warp_hist[kWarps][kRadix];
    uint32_t digit_start[kRadix];
    uint32_t scan_tmp[kWarps];
    uint32_t red[kWarps][6];
    uint64_t kred[kWarps][3];
    uint32_t next;
};

// Tile `tile`'s records [a, a + len) and whether its output goes to
// keys_alt (a chunk whose segment's merge rounds end in keys_out); false
// for an empty tile.
SR_DEV bool tile_span(const TileTables& u, uint32_t tile, uint32_t n_cap, uint32_t& a, uint32_t& len, bool& to_alt) {
    const uint4 d = u.desc[tile];
    uint32_t e;
    to_alt = false;
    if (d.z & kChunkBit) {
        const uint32_t k = d.z & 0xFFFFu, rounds = (d.z >> 16) & 0x7FFFu;
        a = d.x + k * (uint32_t)kTile;
        e = min(a + (uint32_t)kTile, d.x + d.y);
        to_alt = (rounds & 1u) != 0;
    } else {
        a = d.x;
        e = u.tile_end[tile];
    }
    // a frame whose records overflowed the buffers is redone: never read past them
    a = min(a, n_cap);
    e = min(max(e, a), n_cap);
    len = e - a;
    return len > 0 && len <= (uint32_t)kTile;
}

// Stages keys [a, a + len) in buf: [a & ~1, e & ~1) by one bulk copy, key
// e - 1 by a load when e is odd.  Returns the slot of key a (0 or 1), or -1
// when the copy wait gave up (uniform over the CTA, which then leaves).
template <int THREADS>
SR_DEV int stage_tile(uint64_t* buf, uint64_t* bar, uint32_t& phase, const uint64_t* __restrict__ keys_in,
                      uint32_t a, uint32_t len, uint32_t* status, uint32_t spin_limit) {
    const uint32_t e = a + len;
    if ((reinterpret_cast<uintptr_t>(keys_in) & 15u) != 0) {
        for (uint32_t j = threadIdx.x; j < len; j += THREADS) buf[j] = keys_in[a + j];
        __syncthreads();
        return 0;
    }
    const uint32_t a0 = a & ~1u, e0 = e & ~1u;
    const uint32_t nb = e0 - a0;   // e > a >= a0, so e0 >= a0
    if (threadIdx.x == 0) {
        if (nb) {
            // the previous tile's reads of the buffer came before (the
            // caller's barrier); order them before the copy's writes
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            mbar_expect_tx(bar, nb * 8u);
            bulk_load(buf, keys_in + a0, nb * 8u, bar);
        }
        if (e & 1u) buf[nb] = keys_in[e - 1];
    }
    __syncthreads();
    const bool ok = nb == 0 || mbar_wait_bounded(bar, phase, spin_limit, status);
    if (__syncthreads_or(!ok)) {
        // gave up: let the copy land before the CTA leaves, whatever limit it
        // was that the wait ran into
        if (nb) mbar_wait_bounded(bar, phase, max(spin_limit, kSpinLimitDefault), nullptr);
        return -1;
    }
    if (nb) phase ^= 1u;
    return (int)(a - a0);
}

// Field ranges of a tile, reduced over the CTA (every thread gets them).
struct Ranges {
    uint32_t pmin, pmax, rmin, rmax, xmin, xmax;
    uint64_t lo, hi, top;   // key bits' min and max, whole key's max
    SR_DEV void init() {
        pmin = rmin = xmin = ~0u;
        pmax = rmax = xmax = 0;
        lo = ~0ull;
        hi = top = 0;
    }
    SR_DEV void add(const KeyFields& kf, uint64_t k, uint64_t kmask) {
        const uint32_t p = kf.p(k), r = kf.r(k), x = kf.x(k);
        pmin = min(pmin, p); pmax = max(pmax, p);
        rmin = min(rmin, r); rmax = max(rmax, r);
        xmin = min(xmin, x); xmax = max(xmax, x);
        lo = min(lo, k & kmask);
        hi = max(hi, k & kmask);
        top = max(top, k);
    }
    SR_DEV void reduce(PassSmem& S) {
        const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            pmin = min(pmin, __shfl_xor_sync(0xFFFFFFFFu, pmin, o));
            pmax = max(pmax, __shfl_xor_sync(0xFFFFFFFFu, pmax, o));
            rmin = min(rmin, __shfl_xor_sync(0xFFFFFFFFu, rmin, o));
            rmax = max(rmax, __shfl_xor_sync(0xFFFFFFFFu, rmax, o));
            xmin = min(xmin, __shfl_xor_sync(0xFFFFFFFFu, xmin, o));
            xmax = max(xmax, __shfl_xor_sync(0xFFFFFFFFu, xmax, o));
            lo = min(lo, __shfl_xor_sync(0xFFFFFFFFu, lo, o));
            hi = max(hi, __shfl_xor_sync(0xFFFFFFFFu, hi, o));
            top = max(top, __shfl_xor_sync(0xFFFFFFFFu, top, o));
        }
        if (lane == 0) {
            S.red[warp][0] = pmin; S.red[warp][1] = pmax;
            S.red[warp][2] = rmin; S.red[warp][3] = rmax;
            S.red[warp][4] = xmin; S.red[warp][5] = xmax;
            S.kred[warp][0] = lo; S.kred[warp][1] = hi; S.kred[warp][2] = top;
        }
        __syncthreads();
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            pmin = min(pmin, S.red[w][0]); pmax = max(pmax, S.red[w][1]);
            rmin = min(rmin, S.red[w][2]); rmax = max(rmax, S.red[w][3]);
            xmin = min(xmin, S.red[w][4]); xmax = max(xmax, S.red[w][5]);
            lo = min(lo, S.kred[w][0]); hi = max(hi, S.kred[w][1]); top = max(top, S.kred[w][2]);
        }
    }
};

// The minima of the fields and their widths, read back from the
// reduction's shared words (fewer live registers through the passes).
struct Unpack {
    uint32_t pmin, rmin, xmin, rb, xb;
    SR_DEV void load(const PassSmem& S) {
        uint32_t r1 = S.red[0][3], x1 = S.red[0][5];
        pmin = S.red[0][0];
        rmin = S.red[0][2];
        xmin = S.red[0][4];
#pragma unroll
        for (int w = 1; w < kWarps; ++w) {
            pmin = min(pmin, S.red[w][0]);
            rmin = min(rmin, S.red[w][2]); r1 = max(r1, S.red[w][3]);
            xmin = min(xmin, S.red[w][4]); x1 = max(x1, S.red[w][5]);
        }
        rb = bits_of(r1 - rmin);
        xb = bits_of(x1 - xmin);
    }
    // the key of compact fields c
    SR_DEV uint64_t key(const KeyFields& kf, uint32_t c) const {
        const uint32_t x = xmin + (c & low_mask(xb));
        const uint32_t r = rmin + (uint32_t)(((uint64_t)c >> xb) & low_mask(rb));
        const uint32_t p = pmin + (uint32_t)((uint64_t)c >> (rb + xb));
        return ((uint64_t)p << (kf.xb + kf.rb)) | ((uint64_t)r << kf.xb) | (uint64_t)x;
    }
};

// Ranges of a tile's fields, with the row ranks compacted: the ranks in use
// below the off-canvas rank (a band), then the off-canvas rank, then row 0's
// rank above it take consecutive codes, so a tile holding off-canvas or row-0
// records does not need the whole rank range.  Off-canvas records have x 0
// (how keys are packed) and do not widen the x range.  The order of the codes
// is the order of the ranks, and equal keys keep equal codes.
struct TileRanges {
    uint32_t pmin, pmax, bmin, bmax, xmin, xmax, pay_max;
    uint32_t flags;   // kHasOff | kHasTop | kOffX
    static constexpr uint32_t kHasOff = 1, kHasTop = 2, kOffX = 4;
    SR_DEV void init() {
        pmin = bmin = xmin = ~0u;
        pmax = bmax = xmax = pay_max = flags = 0;
    }
    SR_DEV void add(const KeyFields& kf, uint64_t k) {
        const uint32_t p = kf.p(k), r = kf.r(k), x = kf.x(k);
        pmin = min(pmin, p); pmax = max(pmax, p);
        if (r == kf.off_rank) {
            flags |= x ? kHasOff | kOffX : kHasOff;
        } else {
            if (r < kf.off_rank) {
                bmin = min(bmin, r); bmax = max(bmax, r);
            } else {
                flags |= kHasTop;
            }
            xmin = min(xmin, x); xmax = max(xmax, x);
        }
        pay_max = max(pay_max, kf.pay(k));
    }
    // over the CTA's warps, through red[warps][8] (a barrier inside)
    template <int WARPS> SR_DEV void reduce(uint32_t (*red)[8]) {
        static_assert(WARPS <= 32, "a lane a warp");
        const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
        warp_reduce();
        if (lane == 0) {
            uint32_t* w = red[warp];
            w[0] = pmin; w[1] = pmax; w[2] = bmin; w[3] = bmax;
            w[4] = xmin; w[5] = xmax; w[6] = pay_max; w[7] = flags;
        }
        __syncthreads();
        init();
        if (lane < WARPS) {
            const uint32_t* w = red[lane];
            pmin = w[0]; pmax = w[1]; bmin = w[2]; bmax = w[3];
            xmin = w[4]; xmax = w[5]; pay_max = w[6]; flags = w[7];
        }
        warp_reduce();
    }
    SR_DEV void warp_reduce() {
        constexpr uint32_t all = 0xFFFFFFFFu;
        pmin = __reduce_min_sync(all, pmin); pmax = __reduce_max_sync(all, pmax);
        bmin = __reduce_min_sync(all, bmin); bmax = __reduce_max_sync(all, bmax);
        xmin = __reduce_min_sync(all, xmin); xmax = __reduce_max_sync(all, xmax);
        pay_max = __reduce_max_sync(all, pay_max); flags = __reduce_or_sync(all, flags);
    }
    SR_DEV uint32_t has_off() const { return flags & kHasOff; }
    SR_DEV uint32_t has_top() const { return (flags & kHasTop) >> 1; }
    SR_DEV uint32_t band() const { return bmin <= bmax ? bmax - bmin + 1u : 0u; }
    SR_DEV uint32_t rank_codes() const { return band() + has_off() + has_top(); }
    SR_DEV uint32_t bits_p() const { return bits_of(pmax - pmin); }
    SR_DEV uint32_t bits_r() const { return bits_of(rank_codes() - 1u); }
    SR_DEV uint32_t bits_x() const { return xmin <= xmax ? bits_of(xmax - xmin) : 0u; }
    // compact fields of key k (br, bx: bits_r(), bits_x())
    SR_DEV uint32_t code(const KeyFields& kf, uint64_t k, uint32_t br, uint32_t bx) const {
        const uint32_t p = kf.p(k), r = kf.r(k), x = kf.x(k);
        const uint32_t nb = band();
        const bool off = r == kf.off_rank;
        const uint32_t rc = r < kf.off_rank ? r - bmin : (off ? nb : nb + has_off());
        const uint32_t xc = off ? 0u : x - xmin;
        const uint32_t pc = bits_p() ? (p - pmin) << (br + bx) : 0u;
        return pc | (br ? rc << bx : 0u) | xc;
    }
    // the key of compact fields c
    SR_DEV uint64_t key(const KeyFields& kf, uint32_t c, uint32_t br, uint32_t bx) const {
        const uint32_t xc = c & low_mask(bx);
        const uint32_t rc = (uint32_t)(((uint64_t)c >> bx) & low_mask(br));
        const uint32_t p = pmin + (uint32_t)((uint64_t)c >> (br + bx));
        const uint32_t nb = band();
        const uint32_t r = rc < nb ? bmin + rc : (has_off() && rc == nb ? kf.off_rank : kf.off_rank + 1u);
        const uint32_t x = r == kf.off_rank ? 0u : xmin + xc;
        return ((uint64_t)p << (kf.xb + kf.rb)) | ((uint64_t)r << kf.xb) | (uint64_t)x;
    }
};

// `passes` digit passes over items buf[cur][0, len), each into the other
// buffer; returns the buffer holding the result.  digit(item, shift).  hist:
// a histogram of 1 << BITS counts a warp.
template <typename T, int THREADS, int BITS, typename H, typename Digit>
SR_DEV uint32_t radix_passes(H* hist, uint32_t* digit_start, uint32_t* scan_tmp, T* buf0, T* buf1, uint32_t cur,
                             uint32_t len, uint32_t passes, Digit digit) {
    constexpr int kWarps = THREADS / 32, kItems = kTile / THREADS, kRadix = 1 << BITS, kRadixBits = BITS;
    constexpr int kDigitsPerThread = kRadix > THREADS ? kRadix / THREADS : 1;
    const uint32_t tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
    const uint32_t wfirst = warp * (32u * kItems);
    const uint32_t rows = wfirst >= len ? 0u : min((uint32_t)kItems, (len - wfirst + 31u) / 32u);
    for (uint32_t pass = 0; pass < passes; ++pass) {
        const uint32_t shift = pass * kRadixBits;
        const T* in = cur ? buf1 : buf0;
        T* out = cur ? buf0 : buf1;
        for (int i = tid; i < kWarps * kRadix; i += THREADS) hist[i] = 0;
        __syncthreads();
        // rank within the warp: warp w holds slots [w*512, w*512 + 512)
        uint32_t rd[kItems];   // rank | digit << 16
#pragma unroll
        for (int it = 0; it < kItems; ++it) {
            if ((uint32_t)it >= rows) break;
            const uint32_t j = wfirst + (uint32_t)it * 32u + lane;
            const bool ok = j < len;
            const uint32_t dg = ok ? digit(in[j], shift) : (uint32_t)kRadix;
            // (tiles hold runs of nearly sorted keys: a warp sees few digits)
            const uint32_t peers = __match_any_sync(0xFFFFFFFFu, dg);
            const uint32_t leader = (uint32_t)(__ffs(peers) - 1);
            uint32_t before = 0;
            if (ok && lane == leader) {
                before = hist[warp * kRadix + dg];
                hist[warp * kRadix + dg] = (H)(before + (uint32_t)__popc(peers));
            }
            before = __shfl_sync(0xFFFFFFFFu, before, leader);
            rd[it] = (before + (uint32_t)__popc(peers & lanemask_lt())) | (dg << 16);
            __syncwarp();
        }
        __syncthreads();
        // per digit: exclusive over warps, then over digits (a thread takes
        // kDigitsPerThread adjacent digits)
        static_assert(kDigitsPerThread == 1 || THREADS * kDigitsPerThread == kRadix, "digits per thread");
        uint32_t dcnt[kDigitsPerThread];
        uint32_t cnt = 0;
#pragma unroll
        for (int q = 0; q < kDigitsPerThread; ++q) {
            const uint32_t dd = tid * kDigitsPerThread + (uint32_t)q;
            uint32_t sum = 0;
            if (dd < (uint32_t)kRadix) {
#pragma unroll
                for (int w = 0; w < kWarps; ++w) {
                    const uint32_t c = hist[w * kRadix + dd];
                    hist[w * kRadix + dd] = (H)sum;
                    sum += c;
                }
            }
            dcnt[q] = sum;
            cnt += sum;
        }
        uint32_t x = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
            if ((int)lane >= o) x += y;
        }
        if (lane == 31) scan_tmp[warp] = x;
        __syncthreads();
        if (warp == 0) {
            const uint32_t w = lane < kWarps ? scan_tmp[lane] : 0u;
            uint32_t wi = w;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, wi, o);
                if ((int)lane >= o) wi += y;
            }
            if (lane < kWarps) scan_tmp[lane] = wi - w;
        }
        __syncthreads();
        uint32_t start = scan_tmp[warp] + x - cnt;
#pragma unroll
        for (int q = 0; q < kDigitsPerThread; ++q) {
            const uint32_t dd = tid * kDigitsPerThread + (uint32_t)q;
            if (dd < (uint32_t)kRadix) digit_start[dd] = start;
            start += dcnt[q];
        }
        __syncthreads();
#pragma unroll
        for (int it = 0; it < kItems; ++it) {
            if ((uint32_t)it >= rows) break;
            const uint32_t j = wfirst + (uint32_t)it * 32u + lane;
            const uint32_t dg = rd[it] >> 16;
            if (j < len) out[digit_start[dg] + hist[warp * kRadix + dg] + (rd[it] & 0xFFFFu)] = in[j];
        }
        __syncthreads();
        cur ^= 1u;
    }
    return cur;
}

// ---- the tile sort
// Bins of a tile and where a bin is too full for the search in it.
constexpr int kSortThreads = 512;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortRows = kTile / kSortThreads;
constexpr uint32_t kBins = 4096;
constexpr uint32_t kHeavyBin = 384;
constexpr uint32_t kIndexBits = 12;   // a record's index in its tile
constexpr int kSortBits = 8;          // digits of the radix passes
static_assert(kTile == 1 << kIndexBits && kBins == 8u * kSortThreads && kBins <= 1u << 14,
              "tile geometry: eight bins a thread");

struct TileSmem {
    union {
        uint64_t keys[kTile + 2];        // the staged tile
        uint32_t items[2][kTile + 4];    // radix passes: their buffers, once the keys are read
    };
    union {
        struct {
            uint4 slot4[kTile / 4];      // low code << 12 | index, bin by bin; before, a path's first off-canvas place
            uint4 bins4[kBins / 8];      // two 16-bit counts a word; then the bins' starts
            uint16_t slot_bin[kTile];    // bin | kOffSlot of a slot
        };
        struct {
            uint16_t hist[kSortWarps * (1 << kSortBits)];
            uint32_t digit_start[1 << kSortBits];
        };
    };
    uint32_t red[kSortWarps][8];
    uint32_t warp_off[kSortWarps];   // off-canvas records of a warp
    uint32_t scan_tmp[kSortWarps];
    TileRanges ranges;
    uint64_t bar;
    uint32_t next;
    bool grouped;   // the records are grouped by path
};
constexpr uint16_t kOffSlot = 1u << 14;

// How a tile's records fall into bins: `stride` bins a path, `band` of them
// for its rows on the canvas but row 0 (rank code and x, shifted right), then
// one for its off-canvas records and one for row 0.
struct BinPlan {
    uint32_t stride, band, shift;
    bool ok;
    SR_DEV BinPlan(const TileRanges& R, uint32_t bx) {
        const uint32_t paths = R.pmax - R.pmin + 1u;
        const uint32_t per_path = paths < kBins ? (kBins - 1u) / paths : 0u;   // one bin more holds the end
        const uint32_t nb = R.band();
        band = shift = 0;
        ok = per_path >= 3u && paths <= (uint32_t)kTile;
        if (ok && nb) {
            const uint32_t most = per_path - 2u, last = (nb << bx) - 1u;
            const uint32_t lb = bits_of(last), fl = 31u - (uint32_t)__clz((int)most);
            shift = lb > fl + 1u ? lb - fl - 1u : 0u;
            while ((last >> shift) >= most) ++shift;
            band = (last >> shift) + 1u;
        }
        stride = band + 2u;
        ok = ok && shift <= 32u - kIndexBits && bx <= 32u - kIndexBits;
    }
};

// The tile's records in order, by bins: false when a bin is too full.  The
// records are grouped by path (an off-canvas record's place counts on it).
SR_DEV bool sort_by_bins(TileSmem& S, const TileRanges& R, const BinPlan& B, uint32_t bx, uint32_t base, uint32_t len,
                         const KeyFields& kf, uint64_t* __restrict__ out) {
    const uint32_t tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
    const uint32_t rows = (len + kSortThreads - 1) / kSortThreads;
    const uint32_t wfirst = warp * rows * 32u;
    uint32_t* slot = reinterpret_cast<uint32_t*>(S.slot4);
    uint32_t* bins = reinterpret_cast<uint32_t*>(S.bins4);
    // ---- counts: each record's bin, its place in it (as the counts go, in no
    // order) and the code that orders it there.  An off-canvas record's place
    // among its path's is by index: its rank among the tile's off-canvas
    // records (as warp << 12 | rank in the warp, until the warps' counts are
    // known) less the first one's of its path.
    uint32_t at[kSortRows], low[kSortRows];   // bin | off << 14 | place << 16; low code (off canvas: path)
    uint32_t n_off = 0;
    bool heavy = false;
#pragma unroll
    for (int it = 0; it < kSortRows; ++it) {
        if ((uint32_t)it >= rows) break;
        const uint32_t j = wfirst + (uint32_t)it * 32u + lane;
        const bool live = j < len;
        uint32_t bin = 0, place = 0;
        bool off = false;
        low[it] = 0;
        if (live) {
            const uint64_t k = S.keys[base + j];
            const uint32_t r = kf.r(k), x = kf.x(k);
            const uint32_t path = kf.p(k) - R.pmin;
            bin = path * B.stride;
            off = r == kf.off_rank;
            if (r < kf.off_rank) {
                const uint32_t c = ((r - R.bmin) << bx) | (x - R.xmin);
                bin += c >> B.shift;
                low[it] = c & ((1u << B.shift) - 1u);
            } else {
                bin += B.band + (off ? 0u : 1u);
                low[it] = off ? path : x - R.xmin;
            }
        }
        const uint32_t om = __ballot_sync(0xFFFFFFFFu, off);
        if (om) {
            if (off) place = (warp << kIndexBits) | (n_off + (uint32_t)__popc(om & lanemask_lt()));
            n_off += (uint32_t)__popc(om);
            uint32_t left = om;
            while (left) {   // one path's at a time; mostly there is one
                const int leader = __ffs(left) - 1;
                const uint32_t lbin = __shfl_sync(0xFFFFFFFFu, bin, leader);
                const uint32_t peers = __ballot_sync(0xFFFFFFFFu, off && bin == lbin);
                if ((int)lane == leader) {
                    atomicAdd(&bins[bin >> 1], (uint32_t)__popc(peers) << (16u * (bin & 1u)));
                    atomicMin(&slot[low[it]], place);
                }
                left &= ~peers;
            }
        }
        if (live && !off) {
            const uint32_t sh = 16u * (bin & 1u);
            place = (atomicAdd(&bins[bin >> 1], 1u << sh) >> sh) & 0xFFFFu;
            heavy = heavy || place >= kHeavyBin;
        }
        at[it] = bin | (off ? (uint32_t)kOffSlot : 0u) | (place << 16);
    }
    if (lane == 0) S.warp_off[warp] = n_off;
    if (__syncthreads_or(heavy)) return false;
    // ---- the bins' starts over their counts, eight bins a thread
    const uint4 w = S.bins4[tid];
    const uint32_t two = w.x + w.y + w.z + w.w;   // no half carries: a tile's records
    const uint32_t sum = (two & 0xFFFFu) + (two >> 16);
    const uint32_t wsum = __reduce_add_sync(0xFFFFFFFFu, sum);
    if (lane == 0) S.scan_tmp[warp] = wsum;
    if (R.has_off()) {
        // lane v: off-canvas records of the warps before v
        uint32_t before = lane < kSortWarps ? S.warp_off[lane] : 0u;
        const uint32_t own = before;
#pragma unroll
        for (int o = 1; o < kSortWarps; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, before, o);
            if ((int)lane >= o) before += y;
        }
        before -= own;
        const uint32_t mine = __shfl_sync(0xFFFFFFFFu, before, warp);
#pragma unroll
        for (int it = 0; it < kSortRows; ++it) {
            if ((uint32_t)it >= rows) break;
            const bool off = (at[it] & kOffSlot) != 0;
            const uint32_t first = off ? slot[low[it]] : 0u;
            const uint32_t before_first = __shfl_sync(0xFFFFFFFFu, before, first >> kIndexBits);
            if (off) {
                constexpr uint32_t m = (1u << kIndexBits) - 1u;
                const uint32_t place = mine + ((at[it] >> 16) & m) - before_first - (first & m);
                at[it] = (at[it] & 0xFFFFu) | (place << 16);
            }
        }
    }
    __syncthreads();
    {
        const uint32_t wstart = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? S.scan_tmp[lane] : 0u);
        uint32_t incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if ((int)lane >= o) incl += y;
        }
        const uint32_t c4[4] = {w.x, w.y, w.z, w.w};
        uint32_t s4[4], at0 = wstart + incl - sum;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t second = at0 + (c4[i] & 0xFFFFu);
            s4[i] = at0 | (second << 16);
            at0 = second + (c4[i] >> 16);
        }
        S.bins4[tid] = make_uint4(s4[0], s4[1], s4[2], s4[3]);
    }
    __syncthreads();
    // ---- records to their bins
    const uint16_t* start = reinterpret_cast<const uint16_t*>(S.bins4);
#pragma unroll
    for (int it = 0; it < kSortRows; ++it) {
        if ((uint32_t)it >= rows) break;
        const uint32_t j = wfirst + (uint32_t)it * 32u + lane;
        if (j < len) {
            const uint32_t p = start[at[it] & (kBins - 1u)] + (at[it] >> 16);
            slot[p] = (low[it] << kIndexBits) | j;
            S.slot_bin[p] = (uint16_t)(at[it] & (kBins - 1u + kOffSlot));
        }
    }
    __syncthreads();
    // ---- a slot a thread: its record's rank in its bin (code, then index),
    // counted; its key goes from the staged tile straight to its place.  The
    // lanes of a warp read the same few bins and write next to each other.
    for (uint32_t q = tid; q < len; q += kSortThreads) {
        const uint32_t v = slot[q], b = S.slot_bin[q];
        uint32_t pos = q;
        if (!(b & kOffSlot)) {
            const uint32_t s0 = start[b], s1 = start[b + 1];
            pos = s0;
            for (uint32_t i = s0; i < s1; ++i) pos += slot[i] < v ? 1u : 0u;
        }
        out[pos] = S.keys[base + (v & ((1u << kIndexBits) - 1u))];
    }
    return true;
}

// The same by radix passes over 32-bit items (payload above the compact
// fields): the tiles with a crowded bin, or of too many paths for bins.
SR_DEV void sort_by_digits(TileSmem& S, const TileRanges& R, uint32_t base, uint32_t len, const KeyFields& kf,
                           uint64_t* __restrict__ out) {
    const uint32_t tid = threadIdx.x;
    const uint32_t kbits = kf.kbits();
    const uint32_t br = R.bits_r(), bx = R.bits_x(), bits = R.bits_p() + br + bx;
    if (tid == 0) S.ranges = R;
    // a field shifts only when it is not empty, so no shift reaches 32; through
    // registers: the items overwrite the staged keys
    uint32_t iv[kSortRows];
#pragma unroll
    for (int i = 0; i < kSortRows; ++i) {
        const uint32_t j = tid + (uint32_t)i * kSortThreads;
        iv[i] = 0;
        if (j < len) {
            const uint64_t k = S.keys[base + j];
            iv[i] = (bits < 32u ? kf.pay(k) << bits : 0u) | R.code(kf, k, br, bx);
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kSortRows; ++i) {
        const uint32_t j = tid + (uint32_t)i * kSortThreads;
        if (j < len) S.items[0][j] = iv[i];
    }
    const uint32_t cmask = low_mask(bits);
    const uint32_t passes = (bits + kSortBits - 1) / kSortBits;
    const uint32_t cur = radix_passes<uint32_t, kSortThreads, kSortBits, uint16_t>(
        S.hist, S.digit_start, S.scan_tmp, S.items[0], S.items[1], 0u, len, passes,
        [cmask](uint32_t v, uint32_t shift) -> uint32_t { return ((v & cmask) >> shift) & ((1u << kSortBits) - 1u); });
    const TileRanges U = S.ranges;   // read back: fewer live registers through the passes
    const uint32_t ubr = U.bits_r(), ubx = U.bits_x(), ubits = U.bits_p() + ubr + ubx;
    const uint32_t umask = low_mask(ubits);
    for (uint32_t j = tid; j < len; j += kSortThreads) {
        const uint32_t v = S.items[cur][j];
        const uint64_t pay = ubits < 32u ? (uint64_t)(v >> ubits) : 0ull;
        out[j] = (pay << kbits) | U.key(kf, v & umask, ubr, ubx);
    }
}

// Sorts tile `tile`, or hands it to the 64-bit kernel when its compact fields
// and payload do not fit 32 bits (queued in u.fallback).  False when a copy
// wait gave up.
SR_DEV bool sort_tile(TileSmem& S, uint32_t tile, uint32_t& phase, const uint64_t* __restrict__ keys_in,
                      uint64_t* __restrict__ keys_out, uint64_t* __restrict__ keys_alt, const KeyFields& kf,
                      uint32_t n_cap, const TileTables& u, bool wide, uint32_t* status, uint32_t spin_limit) {
    const uint32_t tid = threadIdx.x;
    uint32_t a, len;
    bool to_alt;
    if (!tile_span(u, tile, n_cap, a, len, to_alt)) return true;
    uint64_t* out = (to_alt ? keys_alt : keys_out) + a;
    // (the copy's wait publishes these)
    S.bins4[tid] = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int i = 0; i < kTile / 4 / kSortThreads; ++i)
        S.slot4[tid + (uint32_t)i * kSortThreads] = make_uint4(~0u, ~0u, ~0u, ~0u);
    const int off = stage_tile<kSortThreads>(S.keys, &S.bar, phase, keys_in, a, len, status, spin_limit);
    if (off < 0) return false;
    const uint32_t base = (uint32_t)off;
    TileRanges R;
    R.init();
    for (uint32_t j = tid; j < len; j += kSortThreads) R.add(kf, S.keys[base + j]);
    R.reduce<kSortWarps>(S.red);
    const uint32_t bx = R.bits_x();
    const uint32_t bits = R.bits_p() + R.bits_r() + bx;
    if (bits + bits_of(R.pay_max) > 32u || (R.flags & TileRanges::kOffX)) {
        if (tid == 0) {
            u.fallback[atomicAdd(u.wide_count, 1u)] = tile;
            if (!wide) set_error(status, ERR_CAPACITY);   // k_local_sort is not launched: the frame is redone
        }
        return true;
    }
    if (bits == 0) {   // one key: already in order
        for (uint32_t j = tid; j < len; j += kSortThreads) out[j] = S.keys[base + j];
        return true;
    }
    const BinPlan B(R, bx);
    if (S.grouped && B.ok && sort_by_bins(S, R, B, bx, base, len, kf, out)) return true;
    sort_by_digits(S, R, base, len, kf, out);
    return true;
}

__global__ void __launch_bounds__(kSortThreads, 2) k_tile_sort(const uint64_t* __restrict__ keys_in,
                                                               uint64_t* __restrict__ keys_out,
                                                               uint64_t* __restrict__ keys_alt, KeyFields kf,
                                                               uint32_t n_cap, uint32_t mt, TileTables u, bool wide,
                                                               uint32_t* status, uint32_t spin_limit) {
    wait_for_stream();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TileSmem& S = *reinterpret_cast<TileSmem*>(smem_raw);
    // tiles past the table exist only in a frame whose records overflowed (redone)
    const uint32_t n_tiles = min(u.ctl[kCtlTiles], mt);
    if (threadIdx.x == 0) {
        mbar_init(&S.bar, 1);
        // In a frame whose records overflowed, or whose offsets are wrong, there
        // are records of the frame before between a path's own.  (Read by one
        // thread: other CTAs may set it now.)
        S.grouped = *status == 0u;
    }
    uint32_t phase = 0;
    // the first tiles by the CTAs' numbers: an SM's second CTA takes one only
    // when every SM has one
    for (uint32_t tile = blockIdx.x; tile < n_tiles;) {
        __syncthreads();   // the previous tile is done with the buffers (before the first: the barrier is set up)
        if (threadIdx.x == 0) S.next = gridDim.x + atomicAdd(&u.ctl[kCtlSortNext], 1u);
        if (!sort_tile(S, tile, phase, keys_in, keys_out, keys_alt, kf, n_cap, u, wide, status, spin_limit)) return;
        __syncthreads();
        tile = S.next;
    }
}

// ---- 64-bit items (the tiles k_tile_sort handed over; rare).  The
// passes run between the tile's range of the input array (scratch by now:
// the 32-bit kernel has staged every tile) and of the output, with the
// histograms in static shared memory (the kernel is launched every frame,
// mostly with nothing handed over, so it holds no large buffers).
SR_DEV void sort_tile64(PassSmem& S, uint32_t tile, uint64_t* keys_in, uint64_t* __restrict__ keys_out,
                        uint64_t* __restrict__ keys_alt, const KeyFields& kf, uint32_t n_cap, const TileTables& u) {
    const uint32_t tid = threadIdx.x;
    uint32_t a, len;
    bool to_alt;
    if (!tile_span(u, tile, n_cap, a, len, to_alt)) return;
    uint64_t* src = keys_in + a;
    uint64_t* dst = (to_alt ? keys_alt : keys_out) + a;
    const uint32_t kbits = kf.kbits();
    const uint64_t kmask = (1ull << kbits) - 1ull;
    Ranges R;
    R.init();
    for (uint32_t j = tid; j < len; j += kThreads) R.add(kf, src[j], kmask);
    R.reduce(S);
    const uint32_t bp = bits_of(R.pmax - R.pmin), br = bits_of(R.rmax - R.rmin), bx = bits_of(R.xmax - R.xmin);
    // compact items when the fields fit 32 bits and the payload the other 32
    const bool compact = bp + br + bx <= 32u && (R.top >> kbits) <= 0xFFFFFFFFull;
    const uint32_t bits =
        compact ? bp + br + bx : (R.lo == R.hi ? 0u : 64u - (uint32_t)__clzll((long long)(R.lo ^ R.hi)));
    const uint32_t passes = (bits + kRadixBits - 1) / kRadixBits;
    if (passes == 0) {
        for (uint32_t j = tid; j < len; j += kThreads) dst[j] = src[j];
        return;
    }
    // the items start where the last pass ends in dst (a thread rewrites only
    // its own slots here; the first pass's barrier publishes them)
    uint64_t* first = (passes & 1u) ? src : dst;
    uint64_t* other = (passes & 1u) ? dst : src;
    for (uint32_t j = tid; j < len; j += kThreads) {
        const uint64_t k = src[j];
        const uint64_t c = ((uint64_t)(kf.p(k) - R.pmin) << (br + bx)) | ((uint64_t)(kf.r(k) - R.rmin) << bx) |
                           (uint64_t)(kf.x(k) - R.xmin);
        first[j] = compact ? ((k >> kbits) << 32) | c : k;
    }
    if (compact) {
        radix_passes<uint64_t, kThreads, kRadixBits, uint32_t>(
            &S.warp_hist[0][0], S.digit_start, S.scan_tmp, first, other, 0u, len, passes,
            [](uint64_t v, uint32_t shift) -> uint32_t {
            return ((uint32_t)v >> shift) & (kRadix - 1);
        });
        Unpack U;
        U.load(S);
        for (uint32_t j = tid; j < len; j += kThreads) {
            const uint64_t v = dst[j];
            dst[j] = ((v >> 32) << kbits) | U.key(kf, (uint32_t)v);
        }
    } else {
        radix_passes<uint64_t, kThreads, kRadixBits, uint32_t>(
            &S.warp_hist[0][0], S.digit_start, S.scan_tmp, first, other, 0u, len, passes,
            [kmask](uint64_t v, uint32_t shift) -> uint32_t {
            return (uint32_t)((v & kmask) >> shift) & (kRadix - 1);
        });
    }
}

__global__ void __launch_bounds__(kThreads) k_local_sort(uint64_t* keys_in, uint64_t* __restrict__ keys_out,
                                                         uint64_t* __restrict__ keys_alt, KeyFields kf, uint32_t n_cap,
                                                         TileTables u) {
    wait_for_stream();
    __shared__ PassSmem S;
    const uint32_t n_tiles = *u.wide_count;
    if (n_tiles == 0) return;   // the usual case: nothing handed over
    for (;;) {
        if (threadIdx.x == 0) S.next = atomicAdd(&u.ctl[kCtlFallbackNext], 1u);
        __syncthreads();   // also: the previous tile is done with the histograms
        const uint32_t i = S.next;
        __syncthreads();
        if (i >= n_tiles) break;
        sort_tile64(S, u.fallback[i], keys_in, keys_out, keys_alt, kf, n_cap, u);
    }
}

// ---------------------------------------------------------------- merge ---
// Round `level` of the merge of large segments: runs of width
// W = kTile << level, pairs merged stably (A before B on equal keys).  The
// CTA of a chunk writes that chunk's output range.  A segment needing r
// rounds has its chunks sorted into keys_out (r even) or keys_alt (r odd),
// and each round flips buffer, so its last round lands in keys_out; rounds
// past r do nothing for it.
constexpr int kMergeParts = 4;                   // work items per chunk
constexpr int kMergeOut = kTile / kMergeParts;   // outputs a merge work item writes
constexpr int kMergeItems = kMergeOut / kThreads;
struct MergeSmem {
    uint64_t in[kMergeOut];    // A part then B part of this item's outputs
    uint64_t out[kMergeOut];
    uint32_t split[4];
};

SR_DEV uint32_t merge_split(const uint64_t* A, uint32_t na, const uint64_t* B, uint32_t nb, uint32_t d, uint64_t kmask) {
    // number of A elements among the first d outputs
    uint32_t lo = d > nb ? d - nb : 0u, hi = min(d, na);
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if ((A[mid] & kmask) <= (B[d - 1 - mid] & kmask)) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// The same split found by a whole warp: 32 probes per step.
SR_DEV uint32_t warp_merge_split(const uint64_t* A, uint32_t na, const uint64_t* B, uint32_t nb, uint32_t d,
                                 uint64_t kmask) {
    const uint32_t lane = lane_id();
    uint32_t lo = d > nb ? d - nb : 0u, hi = min(d, na);
    while (lo < hi) {
        const uint32_t step = (hi - lo + 31) / 32;
        const uint32_t m = lo + lane * step;
        const bool valid = m < hi;
        const bool take_a = valid && (A[m] & kmask) <= (B[d - 1 - m] & kmask);
        const uint32_t ta = (uint32_t)__popc(__ballot_sync(0xFFFFFFFFu, take_a));
        const uint32_t tv = (uint32_t)__popc(__ballot_sync(0xFFFFFFFFu, valid));
        // the predicate holds for the first ta probes and fails from probe ta on
        const uint32_t new_lo = ta == 0 ? lo : lo + (ta - 1) * step + 1;
        const uint32_t new_hi = ta < tv ? lo + ta * step : hi;
        lo = new_lo;
        hi = new_hi;
    }
    return lo;
}

// Work item w is part w % kMergeParts of the w / kMergeParts-th chunk of the
// segments that still merge in this round (by classes of rounds: with all
// chunks in one list the last round of the 4096^2 frame spent 19 us finding
// that most had nothing to do, 10 now); the CTAs are persistent (one
// wave) and take items from the round's counter.
SR_DEV void merge_item(MergeSmem& S, uint32_t item, uint32_t chunk, uint64_t* __restrict__ keys_out,
                       uint64_t* __restrict__ keys_alt,
                       uint32_t level, uint32_t key_bits, uint32_t n_cap, const TileTables& u) {
    const uint4 desc = u.desc[chunk];
    const uint32_t k = desc.z & 0xFFFFu, rounds = (desc.z >> 16) & 0x7FFFu;
    if (level >= rounds) return;
    const uint64_t* src = ((rounds - level) & 1u) ? keys_alt : keys_out;
    uint64_t* dst = ((rounds - level) & 1u) ? keys_out : keys_alt;
    const uint32_t s0 = desc.x, size = desc.y;
    if ((uint64_t)s0 + size > n_cap) return;   // overflowed frame: redone
    const uint32_t o0 = k * (uint32_t)kTile + (item % kMergeParts) * (uint32_t)kMergeOut;
    if (o0 >= size) return;
    const uint32_t o1 = min(o0 + (uint32_t)kMergeOut, size);
    const uint32_t W = (uint32_t)kTile << level;
    const uint32_t p0 = (o0 / (2 * W)) * (2 * W);
    const uint32_t na = min(W, size - p0);
    const uint32_t nb = size - p0 > W ? min(W, size - p0 - W) : 0u;
    const uint64_t* A = src + s0 + p0;
    const uint64_t* B = A + na;
    const uint32_t tid = threadIdx.x;
    if (nb == 0) {   // a lone run: already in order
        for (uint32_t j = o0 + tid; j < o1; j += kThreads) dst[s0 + j] = src[s0 + j];
        return;
    }
    const uint64_t kmask = (1ull << key_bits) - 1ull;
    const uint32_t d0 = o0 - p0, d1 = o1 - p0;
    const uint32_t warp = tid >> 5;
    if (warp < 2) {
        const uint32_t sp = warp_merge_split(A, na, B, nb, warp == 0 ? d0 : d1, kmask);
        if (lane_id() == 0) S.split[warp] = sp;
    }
    __syncthreads();
    // (Of sorted runs the second split is not below the first, nor further on
    // than n.  A frame that is redone may merge a chunk that nobody sorted: its
    // parts stay within the runs and the buffers too.)
    const uint32_t n = d1 - d0, ia0 = S.split[0], ia1 = min(max(S.split[1], ia0), ia0 + n);
    const uint32_t ib0 = d0 - ia0, nA = ia1 - ia0, nB = n - nA;
    for (uint32_t j = tid; j < nA; j += kThreads) S.in[j] = A[ia0 + j];
    for (uint32_t j = tid; j < nB; j += kThreads) S.in[nA + j] = B[ib0 + j];
    __syncthreads();
    // each thread merges kItems outputs from its own split
    const uint32_t dt = min(tid * (uint32_t)kMergeItems, n);
    const uint64_t* sA = S.in;
    const uint64_t* sB = S.in + nA;
    uint32_t ia = merge_split(sA, nA, sB, nB, dt, kmask);
    uint32_t ib = dt - ia;
    const uint32_t e = min(dt + (uint32_t)kMergeItems, n);
    for (uint32_t o = dt; o < e; ++o) {
        const bool takeA = ib >= nB || (ia < nA && (sA[ia] & kmask) <= (sB[ib] & kmask));
        S.out[o] = takeA ? sA[ia++] : sB[ib++];
    }
    __syncthreads();
    for (uint32_t j = tid; j < n; j += kThreads) dst[s0 + o0 + j] = S.out[j];
}

__global__ void __launch_bounds__(kThreads) k_merge_level(uint64_t* __restrict__ keys_out,
                                                          uint64_t* __restrict__ keys_alt, uint32_t level,
                                                          uint32_t key_bits, uint32_t n_cap, TileTables u) {
    wait_for_stream();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    MergeSmem& S = *reinterpret_cast<MergeSmem*>(smem_raw);
    __shared__ uint32_t next;
    uint32_t count[kMergeClasses], n_items = 0;
#pragma unroll
    for (uint32_t r = 0; r < kMergeClasses; ++r) {
        count[r] = r >= level ? min(u.ctl[kCtlChunks + 1 + r], u.mt) : 0u;
        n_items += (uint32_t)kMergeParts * count[r];
    }
    for (;;) {
        if (threadIdx.x == 0) next = atomicAdd(&u.ctl[kCtlMergeNext + level], 1u);
        __syncthreads();   // also: the previous item is done with the buffers
        const uint32_t item = next;
        __syncthreads();
        if (item >= n_items) break;
        uint32_t at = item / kMergeParts, cls = 0;
#pragma unroll
        for (uint32_t r = 0; r + 1 < kMergeClasses; ++r)
            if (cls == r && at >= count[r]) {
                at -= count[r];
                cls = r + 1;
            }
        merge_item(S, item, u.chunks[(size_t)cls * u.mt + at], keys_out, keys_alt, level, key_bits, n_cap, u);
    }
}

// ------------------------------------------------------------- launches --
size_t segsort_table_bytes(uint32_t P, int64_t cap) {
    const size_t mt = max_tiles(P, cap);
    return round256(mt * 16) + round256(kMergeClasses * mt * 4) + round256(mt * 4);
}
size_t segsort_zeroed_bytes(uint32_t P, int64_t cap) { return 256 + scan_area(P) + round256(max_tiles(P, cap) * 4); }

int segsort_tile() { return kTile; }

TileTables segsort_tables(const SegArgs& a) { return carve(a); }

cudaError_t segsort_tile_counts(const SegArgs& a, uint32_t out[2]) {
    TileTables u = carve(a);
    cudaError_t e = cudaMemcpy(&out[0], u.ctl + kCtlTiles, 4, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(&out[1], a.wide_count, 4, cudaMemcpyDeviceToHost);
    out[0] = std::min<uint32_t>(out[0], (uint32_t)max_tiles(a.n_paths, a.cap));
    return e;
}

void launch_segsort_largest(const SegArgs& a, cudaStream_t st) {
    if (a.n_paths == 0) return;
    count_launches(1);
    k_seg_largest<<<(a.n_paths + 255) / 256, 256, 0, st>>>(a);
}

void launch_segsort(const SegArgs& sa, uint64_t* keys_in, uint64_t* keys_out, uint64_t* keys_alt, const KeyLayout& L,
                    int levels, int sm_count, uint32_t* status, cudaStream_t st) {
    if (sa.cap <= 0 || sa.n_paths == 0) return;
    TileTables u = carve(sa);
    const size_t mt = max_tiles(sa.n_paths, sa.cap);
    if (!sa.tables_built) {
        count_launches(1);
        launch_after(k_seg_tiles, (sa.n_paths + kSegThreads - 1) / kSegThreads, kSegThreads, 0, st, sa, u, status,
                     spin_limit());
    }
    const uint32_t key_bits = L.pbits + L.rbits + L.xbits;
    const KeyFields kf{L.xbits, L.rbits, L.pbits, (uint32_t)(L.Hy - 1)};
    // resident CTAs per SM of the two persistent kernels (same on every
    // device of the build's architecture)
    static std::atomic<uint32_t> attr{0};
    static std::atomic<int> occ_sort{0}, occ_merge{0};
    once_per_device(attr, [] {
        cudaFuncSetAttribute(k_tile_sort, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TileSmem));
        cudaFuncSetAttribute(k_merge_level, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(MergeSmem));
        int a = 0, c = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, k_tile_sort, kSortThreads, sizeof(TileSmem));
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&c, k_merge_level, kThreads, sizeof(MergeSmem));
        occ_sort.store(std::max(a, 1));
        occ_merge.store(std::max(c, 1));
    });
    const size_t sms = (size_t)std::max(sm_count, 1);
    const unsigned g_tile = (unsigned)std::min<size_t>(mt, sms * (size_t)std::max(occ_sort.load(), 1));
    // the 64-bit sort takes the few tiles the 32-bit one hands over
    const unsigned g_sort = (unsigned)std::min<size_t>(mt, sms);
    const unsigned g_merge =
        (unsigned)std::min<size_t>(kMergeParts * mt, sms * (size_t)std::max(occ_merge.load(), 1));
    count_launches(1 + (sa.wide ? 1 : 0) + (uint32_t)levels);
    const uint32_t n_cap = (uint32_t)sa.cap;
    launch_after(k_tile_sort, g_tile, kSortThreads, sizeof(TileSmem), st, keys_in, keys_out, keys_alt, kf, n_cap,
                 (uint32_t)mt, u, sa.wide, status, spin_limit());
    if (sa.wide) launch_after(k_local_sort, g_sort, kThreads, 0, st, keys_in, keys_out, keys_alt, kf, n_cap, u);
    for (int lv = 0; lv < levels; ++lv)
        launch_after(k_merge_level, g_merge, kThreads, sizeof(MergeSmem), st, keys_out, keys_alt, (uint32_t)lv,
                     key_bits, n_cap, u);
}

}  // namespace sr
