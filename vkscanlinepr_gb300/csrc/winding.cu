// winding.cu — one pass over the sorted records that replaces five reference
// dispatches and two host read-backs:
//   shuffle_fragment.comp:17-26            gather of winding changes
//   naive_scan.comp (scanline_rasterizer.cpp:479-506)   winding scan
//   mark_merged_fragment_and_span.comp:22-93            fragment/span flags
//   naive_scan.comp over 2N flags (scanline_rasterizer.cpp:545-580)
//   gen_merged_fragment_and_span.comp:33-103           draw-list emit
//
// Two launches over tiles of 2048 consecutive sorted records (ITEMS 8; 1024
// with ITEMS 4):
//   k_winding_reduce      each tile's (scene head seen, sum since) pair of
//                         winding changes, a fully parallel read of the keys;
//                         its last CTA scans the tile pairs into each tile's
//                         incoming winding prefix;
//   k_winding_runs        the records' winding scan, fragment and span flags,
//                         and the paint runs at their output slots (one
//                         decoupled look-back over the tiles' run counts).
// k_draw_list writes the reference's draw records, in its order (a record's
// merged fragment, then the span ending at it), when they are read back.  It
// finds flags and centre sums by itself, from whole 64-bit keys: a change of
// rule goes into both (the read-back tests hold them together).
//
// The reference's winding scan is global over its one scene's records
// (scanline_rasterizer.cpp:479-506), so a path whose changes do not sum to
// zero carries into the paths after it.  In a batch of scenes chain A is a
// scan segmented at scene boundaries, so each scene sees exactly the global
// scan it would see alone (with one scene the two are the same).
#include "kernels.h"
#include "scan.cuh"

namespace sr {

namespace {
// a winding tile is THREADS x ITEMS records: 256 x 4 or 256 x 8
constexpr uint64_t kFlagA = 1ull << 62;
constexpr uint64_t kFlagP = 2ull << 62;
constexpr uint64_t kValMask = (1ull << 62) - 1;
constexpr uint64_t kHeadBit = 1ull << 61;   // chain A: the tile holds a scene's first record
// chain B value: merged fragments in bits 31..61, spans in bits 0..30
constexpr int kFragShift = 31;
constexpr uint64_t kSpanMask = (1ull << 31) - 1;

SR_DEV bool rule_pass(uint32_t rule, int32_t wn) {
    // mark_merged_fragment_and_span.comp:82
    return (rule == 0u && wn != 0) || (rule == 1u && (wn & 1) != 0);
}

SR_DEV int32_t sx2(uint32_t v) { return (int32_t)(v << 30) >> 30; }   // 2-bit two's complement

template <typename T> SR_DEV T warp_incl(T v) {
    uint32_t lane = lane_id();
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        T t = __shfl_up_sync(0xFFFFFFFFu, v, d);
        if ((int)lane >= d) v = v + t;
    }
    return v;
}

// Look-back over the tiles' packed counts: a word carries flag and value
// together, so relaxed accesses suffice.
SR_DEV uint64_t lookback(uint64_t* tstat, uint32_t tile, uint32_t* status, uint32_t spin_limit) {
    const uint32_t lane = lane_id();
    uint64_t excl = 0;
    int64_t look = (int64_t)tile - 1;
    uint32_t spins = 0;
    while (look >= 0) {
        const int64_t j = look - (int64_t)lane;
        const uint64_t s = j >= 0 ? ld_relaxed_u64(&tstat[j]) : kFlagP;
        const uint32_t flag = (uint32_t)(s >> 62);
        const uint32_t ready = __ballot_sync(0xFFFFFFFFu, flag != 0);
        const uint32_t pm = __ballot_sync(0xFFFFFFFFu, flag == 2);
        const int firstp = pm ? (__ffs(pm) - 1) : 31;
        const uint32_t need = firstp == 31 ? 0xFFFFFFFFu : ((2u << firstp) - 1u);
        if ((ready & need) != need) {
            if (++spins > spin_limit) {
                if (lane == 0) set_error(status, ERR_LOOKBACK_TIMEOUT);
                break;
            }
            __nanosleep(32);
            continue;
        }
        uint64_t v = ((int)lane <= firstp) ? (s & kValMask) : 0ull;
#pragma unroll
        for (int d = 16; d >= 1; d >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, d);
        excl += v;
        if (pm) break;
        look -= 32;
    }
    return excl;
}

// A tile's draw records in output order, as items of shared memory: the
// record's index in the tile (bits 13..), a span bit (12) and, for a merged
// fragment, its index among the tile's fragments (0..11).  A record gives at
// most a fragment and a span, so 2 x kTile items always fit.
constexpr uint32_t kItemSpan = 1u << 12;
constexpr int kItemRecShift = 13;

template <int ITEMS, int THREADS> struct DrawSmem {
    uint32_t tile;
    int32_t warpA[THREADS / 32];
    int32_t warpAf[THREADS / 32];
    uint32_t warpB[THREADS / 32];
    uint64_t prefixB;
    uint32_t count;
    uint32_t lo_prev;                               // low key half of the record before the tile
    // per thread: the key of its first record, the centre parts of its
    // leading run (records with that key) and whether all its records share it
    uint32_t run_p[THREADS], run_l[THREADS];
    int32_t run_sum[THREADS];
    uint32_t run_all[THREADS];
    uint64_t next_key;                              // the record after the tile, ~0 if none
    int32_t next_c;                                 // its centre part
    uint32_t items[2 * THREADS * ITEMS];
    __align__(16) uint32_t lo[THREADS * ITEMS];     // low key half (row rank, x + 1) of each record
    __align__(16) uint32_t paint[THREADS * ITEMS];  // fill_info of each record's path
};

// Key of record i without its payload, and its packed winding bits.
SR_DEV uint64_t wkey(const WindArgs& a, int64_t i, int64_t n, uint32_t& wb, uint32_t* status) {
    const uint64_t kr = a.skeys[i];
    if (a.svals) {
        const uint32_t rec = a.svals[i];
        if (rec < (uint64_t)n) {
            wb = a.wnp[rec];
        } else {
            wb = 0;
            set_error(status, ERR_BAD_INDEX);
        }
        return kr;
    }
    wb = payload_part(a.L, kr);
    return key_part(a.L, kr);
}

// This thread's ITEMS consecutive records from ibase: keys without their
// payload, and the packed winding bits (4 bits a record).  Records at or past
// n read as key 0; a key whose path is out of range reads as 0 and is flagged.
template <int ITEMS>
SR_DEV void load_run(const WindArgs& a, int64_t ibase, int64_t n, uint64_t (&kk)[ITEMS], uint32_t& wbits,
                     uint32_t* status) {
    const uint32_t pshift = a.L.xbits + a.L.rbits;
    wbits = 0;
    if (!a.svals && ibase + ITEMS <= n) {
        const ulonglong2* p = reinterpret_cast<const ulonglong2*>(a.skeys + ibase);
#pragma unroll
        for (int q = 0; q < ITEMS / 2; ++q) {
            const ulonglong2 v = p[q];
            kk[2 * q] = v.x;
            kk[2 * q + 1] = v.y;
        }
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            wbits |= payload_part(a.L, kk[k]) << (4 * k);
            kk[k] = key_part(a.L, kk[k]);
        }
    } else {
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            uint32_t wb = 0;
            kk[k] = ibase + k < n ? wkey(a, ibase + k, n, wb, status) : 0ull;
            wbits |= (wb & 0xFu) << (4 * k);
        }
    }
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        if (ibase + k < n && (kk[k] >> pshift) >= a.n_paths) {
            set_error(status, ERR_BAD_INDEX);
            kk[k] = 0;
        }
    }
}

// The record before this thread's first (a shuffle, or a load at a warp's
// first lane); 0 before record 0.
template <int ITEMS>
SR_DEV uint64_t prev_key(const WindArgs& a, int64_t ibase, int64_t n, const uint64_t (&kk)[ITEMS]) {
    uint64_t kp = __shfl_up_sync(0xFFFFFFFFu, kk[ITEMS - 1], 1);
    if (lane_id() == 0) {
        uint32_t wb;
        kp = ibase > 0 && ibase - 1 < n ? wkey(a, ibase - 1, n, wb, nullptr) : 0ull;
        if ((kp >> (a.L.xbits + a.L.rbits)) >= a.n_paths) kp = 0;
    }
    return kp;
}

// Scene heads among this thread's records (bit k: record ibase + k is the
// first record of a scene) and the thread's (head seen, sum since) pair.
template <int ITEMS>
SR_DEV uint32_t run_heads(const WindArgs& a, int64_t ibase, int64_t n, const uint64_t (&kk)[ITEMS], uint64_t kprev,
                          uint32_t wbits, bool& tf, int32_t& tv) {
    const uint32_t pshift = a.L.xbits + a.L.rbits;
    const bool multi = a.st.n_scenes > 1;
    uint32_t heads = 0;
    tf = false;
    tv = 0;
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const int64_t i = ibase + k;
        if (i >= n) continue;
        bool h = i == 0;
        if (multi && !h) {
            const uint64_t kp = k == 0 ? kprev : kk[k - 1];
            h = a.st.path_scene[(uint32_t)(kk[k] >> pshift)] != a.st.path_scene[(uint32_t)(kp >> pshift)];
        }
        if (h) {
            heads |= 1u << k;
            tf = true;
            tv = 0;
        }
        tv = wadd(tv, sx2(wbits >> (4 * k)));
    }
    return heads;
}

// (fa, va) then (fb, vb), into (fb, vb): a head in the second part restarts
// the sum.
SR_DEV void seg_combine(bool fa, int32_t va, bool& fb, int32_t& vb) {
    vb = fb ? vb : wadd(va, vb);
    fb = fb || fa;
}

// Segmented scan of (head, value) pairs over a CTA of THREADS: this
// thread's exclusive pair and the CTA's aggregate.  wv and wf are
// THREADS / 32 words of shared memory each; ends with a barrier.
template <int THREADS>
SR_DEV void cta_seg_scan(bool tf, int32_t tv, int32_t* wv, int32_t* wf, bool& fe, int32_t& ve, bool& aggf,
                         int32_t& agg) {
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    bool fi = tf;
    int32_t vi = tv;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const bool fp = __shfl_up_sync(0xFFFFFFFFu, (int)fi, d) != 0;
        const int32_t vp = __shfl_up_sync(0xFFFFFFFFu, vi, d);
        if ((int)lane >= d) seg_combine(fp, vp, fi, vi);
    }
    bool xf = __shfl_up_sync(0xFFFFFFFFu, (int)fi, 1) != 0;
    int32_t xv = __shfl_up_sync(0xFFFFFFFFu, vi, 1);
    if (lane == 0) {
        xf = false;
        xv = 0;
    }
    if (lane == 31) {
        wv[warp] = vi;
        wf[warp] = fi ? 1 : 0;
    }
    __syncthreads();
    // the warps before this one, and all of them for the aggregate
    bool pf = false;
    int32_t pv = 0;
    aggf = false;
    agg = 0;
#pragma unroll
    for (int w = 0; w < THREADS / 32; ++w) {
        bool f = wf[w] != 0;
        int32_t v = wv[w];
        if (w < (int)warp) {
            bool f2 = f;
            int32_t v2 = v;
            seg_combine(pf, pv, f2, v2);
            pf = f2;
            pv = v2;
        }
        seg_combine(aggf, agg, f, v);
        aggf = f;
        agg = v;
    }
    seg_combine(pf, pv, xf, xv);
    fe = xf;
    ve = xv;
    __syncthreads();
}
}  // namespace

// The tiles' incoming winding prefixes: an exclusive segmented scan of the
// tile pairs by one CTA, eight tiles a thread and round (one a thread took
// 41 rounds, 17 us more, for the 10,290 tiles of a 21 M record frame).  Also
// writes the scan's total (the winding scan's last entry) when the stages are
// kept.
template <int THREADS>
__device__ __noinline__ void scan_tile_pairs(const uint64_t* tagg, int32_t* __restrict__ tile_in, const WindArgs& a, int64_t n,
                            int64_t tiles, int32_t* wv, int32_t* wf) {
    constexpr int K = 8;
    bool cf = false;
    int32_t cv = 0;
    for (int64_t base = 0; base < tiles; base += THREADS * K) {
        const int64_t t = base + (int64_t)threadIdx.x * K;
        uint64_t w[K];
#pragma unroll
        for (int k = 0; k < K; ++k) w[k] = t + k < tiles ? ld_relaxed_u64(&tagg[t + k]) : 0ull;
        bool tf = false;
        int32_t tv = 0;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            bool f = (w[k] & kHeadBit) != 0;
            int32_t v = (int32_t)(uint32_t)w[k];
            seg_combine(tf, tv, f, v);
            tf = f;
            tv = v;
        }
        bool xf, aggf;
        int32_t xv, agg;
        cta_seg_scan<THREADS>(tf, tv, wv, wf, xf, xv, aggf, agg);
        seg_combine(cf, cv, xf, xv);
        // the value since the last head entering each tile, whatever xf says
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (t + k < tiles) tile_in[t + k] = xv;
            bool f = (w[k] & kHeadBit) != 0;
            int32_t v = (int32_t)(uint32_t)w[k];
            seg_combine(xf, xv, f, v);
            xf = f;
            xv = v;
        }
        seg_combine(cf, cv, aggf, agg);
        cf = aggf;
        cv = agg;
    }
    if (threadIdx.x == 0 && a.dbg_wscan) a.dbg_wscan[n] = cv;
}

// Each thread owns ITEMS consecutive sorted records (a blocked layout): its
// keys come in as 16-byte vector loads, the keys on either side of its run
// by warp shuffles (a scalar load at a warp's edges), and the flags stay in
// registers.  The tile's draw records are contiguous in the output, so they
// are listed as items in shared memory and written an item a thread:
// consecutive threads write consecutive records.
template <int ITEMS, int THREADS>
__global__ void __launch_bounds__(THREADS, 4) k_draw_list(const WindArgs a,
                                                              const int32_t* __restrict__ tile_in,
                                                              uint64_t* __restrict__ tstatB, uint32_t* counter,
                                                              uint32_t* status, uint32_t spin_limit) {
    constexpr int kTile = THREADS * ITEMS;
    static_assert(ITEMS % 2 == 0 && ITEMS <= 8, "records per thread");
    static_assert(kTile <= 4096, "record and fragment index of an item");
    __shared__ DrawSmem<ITEMS, THREADS> S;
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) S.tile = atomicAdd(counter, 1u);
    __syncthreads();
    const uint32_t tile = S.tile;
    const int64_t n = a.n_dev ? (int64_t)min((uint64_t)*a.n_dev, (uint64_t)a.n) : a.n;
    const int64_t tbase = (int64_t)tile * kTile;
    if (tbase >= n) return;   // launched for the capacity
    const int32_t t_in = tile_in[tile];
    const uint32_t xbits = a.L.xbits, pshift = a.L.xbits + a.L.rbits;
    const uint32_t xmask = (1u << xbits) - 1u, rmask = (1u << a.L.rbits) - 1u;
    const uint32_t off_rank = (uint32_t)(a.L.Hy - 1);
    const bool multi = a.st.n_scenes > 1;

    // ---- this thread's records: keys and packed winding bits (4 bits each)
    const int64_t ibase = tbase + (int64_t)threadIdx.x * ITEMS;
    const int nvalid = (int)max((int64_t)0, min((int64_t)ITEMS, n - ibase));
    uint64_t kk[ITEMS];
    uint32_t wbits;
    load_run<ITEMS>(a, ibase, n, kk, wbits, status);
    // the fill rule and paint of the first record's path, fetched early
    uint32_t rule_path = nvalid > 0 ? (uint32_t)(kk[0] >> pshift) : 0xFFFFFFFFu;
    uint32_t rule = nvalid > 0 ? a.fill_rule[rule_path] : 0u;
    uint32_t paint_path = rule_path;
    uint32_t paint0 = nvalid > 0 ? a.fill_info[paint_path] : 0u;
    // the record before this thread's first, and after its last
    const uint64_t kprev = prev_key<ITEMS>(a, ibase, n, kk);
    uint64_t knext = __shfl_down_sync(0xFFFFFFFFu, kk[0], 1);
    uint32_t wnext = 0;
    if (lane == 31) knext = ibase + ITEMS < n ? wkey(a, ibase + ITEMS, n, wnext, nullptr) : ~0ull;
    if (nvalid < ITEMS || ibase + ITEMS == n) knext = ~0ull;   // no record after this thread's last
    if (threadIdx.x == THREADS - 1) {
        S.next_key = knext;
        S.next_c = sx2(wnext >> 2);
    }

    // ---- winding prefix: the tile's from the tile scan, then the CTA's
    // segmented scan (segments start at scene heads)
    bool tf, fe, aggf;
    int32_t tv, ve, agg;
    const uint32_t heads = run_heads<ITEMS>(a, ibase, n, kk, kprev, wbits, tf, tv);
    cta_seg_scan<THREADS>(tf, tv, S.warpA, S.warpAf, fe, ve, aggf, agg);
    int32_t wrun = fe ? ve : wadd(t_in, ve);

    // From here a key is handled as two 32-bit halves: its path, and
    // (row rank, x + 1) below it (at most 29 bits for a 16384-pixel canvas).
    // A key is (path, row rank, x + 1) with the rank of an off-canvas record
    // Hy - 1, so two records share a cell exactly when their keys are equal,
    // and a row of one path when they agree above the x bits.
    const uint32_t lomask = (1u << pshift) - 1u;
    uint32_t kp[ITEMS], kl[ITEMS];
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        kp[k] = (uint32_t)(kk[k] >> pshift);
        kl[k] = (uint32_t)kk[k] & lomask;
    }
    const uint32_t pprev = (uint32_t)(kprev >> pshift), lprev = (uint32_t)kprev & lomask;
    {
        uint4* dst = reinterpret_cast<uint4*>(&S.lo[threadIdx.x * ITEMS]);
#pragma unroll
        for (int q = 0; q < ITEMS / 4; ++q) dst[q] = make_uint4(kl[4 * q], kl[4 * q + 1], kl[4 * q + 2], kl[4 * q + 3]);
        if (threadIdx.x == 0) S.lo_prev = lprev;
    }

    // ---- centre parts of each record's cell from it to the cell's end
    // (pixel mode): a reverse segmented sum over runs of equal keys, with
    // the run that continues past this thread walked in global memory
    int32_t csum[ITEMS];
    if (a.pixel_mode) {
        // within the thread
        const bool cont_last = knext == kk[ITEMS - 1];
        csum[ITEMS - 1] = sx2(wbits >> (4 * (ITEMS - 1) + 2));
#pragma unroll
        for (int k = ITEMS - 2; k >= 0; --k) {
            const bool cont = kp[k + 1] == kp[k] && kl[k + 1] == kl[k];
            csum[k] = wadd(sx2(wbits >> (4 * k + 2)), cont ? csum[k + 1] : 0);
        }
        bool all_same = nvalid == ITEMS;
#pragma unroll
        for (int k = 1; k < ITEMS; ++k) all_same = all_same && kp[k] == kp[0] && kl[k] == kl[0];
        S.run_p[threadIdx.x] = kp[0];
        S.run_l[threadIdx.x] = kl[0];
        S.run_sum[threadIdx.x] = csum[0];
        S.run_all[threadIdx.x] = all_same ? 1u : 0u;
        __syncthreads();
        // the run that continues past this thread: the leading runs of the
        // next threads (a thread whose records all share the key passes it
        // on), then the records after the tile.  Only a merged fragment (an
        // on-canvas cell whose run starts in this thread) needs it;
        // off-canvas records of a path share one key (one per row past its
        // right edge) and make long runs, which are never followed.
        const uint32_t pl = kp[ITEMS - 1], ll = kl[ITEMS - 1];
        bool starts_here = pprev != pl || lprev != ll;
#pragma unroll
        for (int k = 1; k < ITEMS; ++k) starts_here = starts_here || kp[k - 1] != pl || kl[k - 1] != ll;
        const uint32_t rankl = (ll >> xbits) & rmask, xol = ll & xmask;
        const uint32_t xo_maxl = (uint32_t)div_F((multi ? scene_of_path(a.st, pl).W : a.W) + a.F - 1, a.F);
        int32_t tail = 0;
        if (cont_last && starts_here && rankl != off_rank && xol >= 1u && xol <= xo_maxl) {
            uint32_t t = threadIdx.x + 1;
            bool follow = true;
            while (follow && t < THREADS) {
                if (S.run_p[t] != pl || S.run_l[t] != ll) {
                    follow = false;
                    break;
                }
                tail = wadd(tail, S.run_sum[t]);
                follow = S.run_all[t] != 0;
                ++t;
            }
            if (follow && S.next_key == kk[ITEMS - 1]) {
                tail = wadd(tail, S.next_c);
                // a run of two or more records past the tile end (rare)
                for (int64_t j = tbase + kTile + 1; j < n; ++j) {
                    uint32_t wb = 0;
                    if (wkey(a, j, n, wb, nullptr) != kk[ITEMS - 1]) break;
                    tail = wadd(tail, sx2(wb >> 2));
                }
            }
        }
        // the last record's run gets the tail, and so do the records before
        // it in the same run
        bool in_run = true;
#pragma unroll
        for (int k = ITEMS - 1; k >= 0; --k) {
            in_run = in_run && kp[k] == pl && kl[k] == ll;
            if (in_run) csum[k] = wadd(csum[k], tail);
        }
    }

    // ---- flags (mark_merged_fragment_and_span.comp:22-93)
    uint32_t ffm = 0, sfm = 0;
    const int32_t F = a.F;
    // on the canvas: a row of it, and 0 <= x = (xo - 1) F < W, i.e. 1 <= xo <= ceil(W / F)
    const uint32_t xo_max1 = (uint32_t)div_F(a.W + F - 1, F);
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        if ((heads >> k) & 1u) wrun = 0;
        const int32_t wscan = wrun;
        wrun = wadd(wrun, sx2(wbits >> (4 * k)));
        if (k >= nvalid) continue;
        const uint32_t p1 = kp[k], l1 = kl[k];
        const uint32_t p0 = k == 0 ? pprev : kp[k - 1], l0 = k == 0 ? lprev : kl[k - 1];
        const uint32_t xo1 = l1 & xmask, rank1 = l1 >> xbits;
        const uint32_t xo_max = multi ? (uint32_t)div_F(scene_of_path(a.st, p1).W + F - 1, F) : xo_max1;
        const bool on = rank1 != off_rank && xo1 >= 1u && xo1 <= xo_max;
        const bool first = ibase + k == 0;
        const bool head = first || p0 != p1 || l0 != l1;
        bool ff = on && head;
        bool sf = !first && p0 == p1 && (l0 >> xbits) == rank1 && (l0 & xmask) + 1u < xo1;
        if (sf || (ff && a.pixel_mode)) {
            if (p1 != rule_path) {
                rule = a.fill_rule[p1];
                rule_path = p1;
            }
            if (sf) sf = rule_pass(rule, wscan);
            // centre sample of the merged cell: scan at its first record plus
            // the left-of-centre changes of the cell's pieces
            if (ff && a.pixel_mode) ff = rule_pass(rule, wadd(wscan, csum[k]));
        }
        if (ff || sf) {
            if (p1 != paint_path) {
                paint0 = a.fill_info[p1];
                paint_path = p1;
            }
            S.paint[threadIdx.x * ITEMS + k] = paint0;
        }
        ffm |= (ff ? 1u : 0u) << k;
        sfm |= (sf ? 1u : 0u) << k;
    }

    // ---- output slots.  Within the CTA the counts are packed 16:16 (a tile
    // has at most 2 x 2048 outputs); across tiles 31:31 with a look-back.
    const uint32_t bsum = ((uint32_t)__popc(ffm) << 16) | (uint32_t)__popc(sfm);
    const uint32_t inclB = warp_incl<uint32_t>(bsum);
    if (lane == 31) S.warpB[warp] = inclB;
    __syncthreads();
    if (warp == 0) {
        const uint32_t w = lane < THREADS / 32 ? S.warpB[lane] : 0u;
        const uint32_t wi = warp_incl<uint32_t>(w);
        if (lane < THREADS / 32) S.warpB[lane] = wi - w;
        const uint32_t agg16 = __shfl_sync(0xFFFFFFFFu, wi, THREADS / 32 - 1);
        const uint64_t aggB = ((uint64_t)(agg16 >> 16) << kFragShift) | (uint64_t)(agg16 & 0xFFFFu);
        if (lane == 0) st_relaxed_u64(&tstatB[tile], (tile == 0 ? kFlagP : kFlagA) | aggB);
        uint64_t excl = 0;
        if (tile > 0) {
            excl = lookback(tstatB, tile, status, spin_limit);
            if (lane == 0) st_relaxed_u64(&tstatB[tile], kFlagP | (excl + aggB));
        }
        if (lane == 0) {
            S.prefixB = excl;
            S.count = (agg16 >> 16) + (agg16 & 0xFFFFu);
        }
    }
    __syncthreads();
    // this thread's items: in record order, a record's fragment before its span
    {
        const uint32_t l0 = S.warpB[warp] + (inclB - bsum);
        uint32_t lf = l0 >> 16, slot = lf + (l0 & 0xFFFFu);
        if (ffm | sfm) {
#pragma unroll
            for (int k = 0; k < ITEMS; ++k) {
                const uint32_t rec = (threadIdx.x * ITEMS + k) << kItemRecShift;
                if ((ffm >> k) & 1u) S.items[slot++] = rec | lf++;
                if ((sfm >> k) & 1u) S.items[slot++] = rec | kItemSpan;
            }
        }
    }
    __syncthreads();

    // ---- the draw records (gen_merged_fragment_and_span.comp:33-103), an
    // item a thread, from the key halves and paint staged in shared memory.
    // An emitted record's cell is on the canvas: y = yy F with yy its row
    // (rank Hy is row 0, rank r < Hy - 1 is row r + 1), x = (xo - 1) F.
    const uint64_t tprefix = S.prefixB;
    const uint32_t tile_cnt = S.count;
    const int64_t tile_first = (int64_t)((tprefix >> kFragShift) + (tprefix & kSpanMask));
    const uint64_t frag0 = tprefix >> kFragShift;
    for (uint32_t j = threadIdx.x; j < tile_cnt; j += THREADS) {
        const uint32_t it = S.items[j], r = it >> kItemRecShift;
        const uint32_t l1 = S.lo[r], rank1 = (l1 >> xbits) & rmask;
        const int32_t y = (rank1 == (uint32_t)a.L.Hy ? 0 : (int32_t)rank1 + 1) * F;
        const int32_t x1 = ((int32_t)(l1 & xmask) - 1) * F;
        int4 d;
        if (!(it & kItemSpan)) {
            d = make_int4((int32_t)((uint32_t)y << 16) | x1, F, (int32_t)S.paint[r],
                          (int32_t)(frag0 + (it & (kItemSpan - 1u)) + 1u));
        } else {
            // the span's left cell is the record before it, in the same
            // path and row (a span is never record 0)
            const uint32_t l0 = r > 0 ? S.lo[r - 1] : S.lo_prev;
            const int32_t x0 = imax(0, wadd(((int32_t)(l0 & xmask) - 1) * F, F));
            d = make_int4((int32_t)((uint32_t)y << 16) | x0, x1 - x0, (int32_t)S.paint[r], 0);
        }
        if (tile_first + j < a.draw_capacity) a.draw[tile_first + j] = d;
    }
}

// ------------------------------------------------------------ paint runs --
// What a frame needs of a key: its path and, below it, the row rank and x + 1
// (at most 30 bits), as two 32-bit words, and its winding bits.  No 64-bit
// shift: the halves come out of the key's words by one funnel shift.
struct KeySplit {
    uint32_t pshift, pmask, lomask, pay;
    bool pay_high;
    SR_DEV explicit KeySplit(const KeyLayout& L) {
        pshift = L.xbits + L.rbits;
        pmask = (1u << L.pbits) - 1u;
        lomask = (1u << pshift) - 1u;
        pay = key_bits(L) & 31u;
        pay_high = key_bits(L) >= 32u;
    }
    SR_DEV uint32_t path(uint2 k) const { return __funnelshift_r(k.x, k.y, pshift) & pmask; }
    SR_DEV uint32_t low(uint2 k) const { return k.x & lomask; }
    SR_DEV uint32_t bits(uint2 k) const { return (pay_high ? k.y >> pay : __funnelshift_r(k.x, k.y, pay)) & 0xFu; }
};

// Record i: its path, low half and winding bits.
SR_DEV void split_record(const WindArgs& a, const KeySplit& ks, int64_t i, int64_t n, uint32_t& path, uint32_t& low,
                         uint32_t& wb, uint32_t* status) {
    const uint2 k = *reinterpret_cast<const uint2*>(a.skeys + i);
    path = ks.path(k);
    low = ks.low(k);
    wb = 0;
    if (!a.svals) {
        wb = ks.bits(k);
    } else {
        const uint32_t rec = a.svals[i];
        if (rec < (uint64_t)n) wb = a.wnp[rec] & 0xFu;
        else set_error(status, ERR_BAD_INDEX);
    }
    if (path >= a.n_paths) {
        set_error(status, ERR_BAD_INDEX);
        path = low = 0;
    }
}

// This thread's ITEMS consecutive records from ibase (4 winding bits a
// record).  Records at or past n read as path 0, low 0.
template <int ITEMS>
SR_DEV void load_split(const WindArgs& a, const KeySplit& ks, int64_t ibase, int64_t n, uint32_t (&kp)[ITEMS],
                       uint32_t (&kl)[ITEMS], uint32_t& wbits, uint32_t* status) {
    wbits = 0;
    if (!a.svals && ibase + ITEMS <= n) {
        const uint4* p = reinterpret_cast<const uint4*>(a.skeys + ibase);
        uint4 v[ITEMS / 2];
#pragma unroll
        for (int q = 0; q < ITEMS / 2; ++q) v[q] = p[q];
        bool bad = false;
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            const uint2 w = k & 1 ? make_uint2(v[k / 2].z, v[k / 2].w) : make_uint2(v[k / 2].x, v[k / 2].y);
            kp[k] = ks.path(w);
            kl[k] = ks.low(w);
            wbits |= ks.bits(w) << (4 * k);
            bad = bad || kp[k] >= a.n_paths;
        }
        if (bad) {
            set_error(status, ERR_BAD_INDEX);
#pragma unroll
            for (int k = 0; k < ITEMS; ++k)
                if (kp[k] >= a.n_paths) kp[k] = kl[k] = 0;
        }
        return;
    }
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        kp[k] = kl[k] = 0;
        if (ibase + k >= n) continue;
        uint32_t wb;
        split_record(a, ks, ibase + k, n, kp[k], kl[k], wb, status);
        wbits |= wb << (4 * k);
    }
}

// Sum of the winding changes (-1, 0 or 1 in the low two of each four bits).
SR_DEV int32_t change_sum(uint32_t wbits) {
    const uint32_t odd = wbits & 0x11111111u, neg = odd & (wbits >> 1);
    return __popc(odd) - 2 * __popc(neg);
}

// Records of this thread that are the first of a scene (bit k).
template <int ITEMS>
SR_DEV uint32_t scene_heads(const WindArgs& a, int64_t ibase, int nvalid, const uint32_t (&kp)[ITEMS], uint32_t pprev) {
    uint32_t heads = 0;
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        if (k >= nvalid) continue;
        const uint32_t p0 = k == 0 ? pprev : kp[k - 1];
        if (ibase + k == 0 || (kp[k] != p0 && a.st.path_scene[kp[k]] != a.st.path_scene[p0])) heads |= 1u << k;
    }
    return heads;
}

// Exclusive prefix of this thread's winding changes in its CTA, and the CTA's
// (head seen, sum since) pair.  Only a batch has heads but record 0, before
// which there is nothing.
template <int THREADS, bool MULTI>
SR_DEV void winding_prefix(uint32_t heads, uint32_t wbits, int32_t* wv, int32_t* wf, bool& fe, int32_t& ve, bool& aggf,
                           int32_t& agg) {
    if (MULTI) {
        const uint32_t last = heads ? 31u - (uint32_t)__clz(heads) : 0u;
        const int32_t tv = change_sum(heads ? wbits & (0xFFFFFFFFu << (4 * last)) : wbits);
        cta_seg_scan<THREADS>(heads != 0, tv, wv, wf, fe, ve, aggf, agg);
        return;
    }
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    const int32_t tv = change_sum(wbits), incl = warp_incl_scan(tv);
    if (lane == 31) wv[warp] = incl;
    __syncthreads();
    int32_t before = 0;
    agg = 0;
#pragma unroll
    for (int w = 0; w < THREADS / 32; ++w) {
        if (w == (int)warp) before = agg;
        agg = wadd(agg, wv[w]);
    }
    ve = wadd(before, incl - tv);
    fe = aggf = false;
    __syncthreads();
}

// Per tile: the (head seen, sum since) pair of its winding changes, a read of
// the keys at DRAM speed: SPLIT warps a tile, 64 records (16 bytes a lane) and
// up to eight loads in flight a round, nothing to wait for but the loads.  A
// scene's head drops what the lanes summed before it.  The CTA that finishes
// last scans the pairs of all tiles (out of line, or its registers would limit
// the CTAs on an SM).  A warp a tile when there are tiles for every SM that
// way; below, a CTA a tile: for 0.37 M records (180 tiles) the kernel and the
// runs after it took 28.6 us with a warp a tile and 24.5 with a CTA; for 21 M
// records 282 and 289.
template <int ITEMS, int THREADS, int SPLIT, bool MULTI>
__global__ void __launch_bounds__(THREADS, 4) k_winding_reduce(const WindArgs a, uint64_t* tagg,
                                                            int32_t* __restrict__ tile_in, uint32_t* done) {
    wait_for_previous();
    constexpr int kTile = 256 * ITEMS, kWarps = THREADS / 32 / SPLIT, kRounds = kTile / 64 / SPLIT;
    constexpr int kFlight = kRounds < 8 ? kRounds : 8;
    static_assert(kRounds % kFlight == 0 && (SPLIT == 1 || kWarps == 1), "a warp a tile, or the CTA's warps");
    __shared__ int32_t wv[THREADS / 32], wf[THREADS / 32];
    __shared__ bool s_last;
    const int64_t n = a.n_dev ? (int64_t)min((uint64_t)*a.n_dev, (uint64_t)a.n) : a.n;
    const int64_t tiles = (n + kTile - 1) / kTile, ctas = (tiles + kWarps - 1) / kWarps;
    if ((int64_t)blockIdx.x >= ctas) return;
    const KeySplit ks(a.L);
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    const int64_t tile = (int64_t)blockIdx.x * kWarps + warp / SPLIT;
    const int64_t tbase = tile * kTile + (warp % SPLIT) * (kTile / SPLIT);
    if (tile < tiles) {
        uint32_t before = 0, l, wb;   // path of the record before the round
        if (MULTI && tbase > 0 && tbase < n) split_record(a, ks, tbase - 1, n, before, l, wb, nullptr);
        bool head = false;
        int32_t sum = 0;
        for (int r0 = 0; r0 < kRounds && tbase + r0 * 64 < n; r0 += kFlight) {
            uint4 v[kFlight];
            const bool vec = !a.svals && tbase + (r0 + kFlight) * 64 <= n;
            if (vec) {
#pragma unroll
                for (int r = 0; r < kFlight; ++r)
                    v[r] = *reinterpret_cast<const uint4*>(a.skeys + tbase + (r0 + r) * 64 + 2 * lane);
            }
#pragma unroll
            for (int r = 0; r < kFlight; ++r) {
                const int64_t i = tbase + (r0 + r) * 64 + 2 * lane;
                const int valid = vec ? 2 : (int)max((int64_t)0, min((int64_t)2, n - i));
                uint32_t p0 = 0, p1 = 0, w0 = 0, w1 = 0;
                if (vec) {
                    const uint2 k0 = make_uint2(v[r].x, v[r].y), k1 = make_uint2(v[r].z, v[r].w);
                    w0 = ks.bits(k0);
                    w1 = ks.bits(k1);
                    p0 = ks.path(k0);
                    p1 = ks.path(k1);
                    if (p0 >= a.n_paths) p0 = 0;
                    if (p1 >= a.n_paths) p1 = 0;
                } else {
                    if (valid > 0) split_record(a, ks, i, n, p0, l, w0, nullptr);
                    if (valid > 1) split_record(a, ks, i + 1, n, p1, l, w1, nullptr);
                }
                int32_t c = change_sum(w0 | (w1 << 4));
                if (MULTI) {
                    uint32_t pl = __shfl_up_sync(0xFFFFFFFFu, p1, 1);
                    if (lane == 0) pl = before;
                    before = __shfl_sync(0xFFFFFFFFu, p1, 31);
                    const bool h0 = valid > 0 && (i == 0 || (p0 != pl && a.st.path_scene[p0] != a.st.path_scene[pl]));
                    const bool h1 = valid > 1 && p1 != p0 && a.st.path_scene[p1] != a.st.path_scene[p0];
                    const uint32_t hm = __ballot_sync(0xFFFFFFFFu, h0 || h1);
                    if (hm) {
                        const uint32_t at = 31u - (uint32_t)__clz(hm);
                        sum = 0;
                        if (lane < at) c = 0;
                        else if (lane == at && h1) c = change_sum(w1);
                        head = true;
                    }
                }
                sum = wadd(sum, c);
            }
        }
        sum = __reduce_add_sync(0xFFFFFFFFu, sum);
        if (lane == 0) {
            if (SPLIT == 1) {
                st_relaxed_u64(&tagg[tile], (head ? kHeadBit : 0ull) | (uint32_t)sum);
                __threadfence();
            } else {
                wv[warp] = sum;
                wf[warp] = head;
            }
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (SPLIT > 1) {
            bool head = false;
            int32_t sum = 0;
            for (int w = 0; w < SPLIT; ++w) {
                sum = wf[w] ? wv[w] : wadd(sum, wv[w]);
                head = head || wf[w];
            }
            st_relaxed_u64(&tagg[tile], (head ? kHeadBit : 0ull) | (uint32_t)sum);
            __threadfence();
        }
        s_last = atomicAdd(done, 1u) == (uint32_t)ctas - 1u;
        __threadfence();
    }
    __syncthreads();
    release_next();
    if (s_last) scan_tile_pairs<THREADS>(tagg, tile_in, a, n, tiles, wv, wf);
}

// Paint runs.  The draw records of one path in one row paint disjoint cells in
// one paint: a merged fragment its cell, a span the cells between two.  Where
// they touch, one run stands for all of them: [first cell, cell after the
// last) of a row.  A simple shape's row is one run instead of a fragment, a
// fragment and a span, so the row sort and the resolve have a third of the
// records to order and to paint.  In a row's order the painted cells and
// gaps come as alternating starts and ends of runs, so the j-th start of a
// tile and the j-th end belong together and are listed independently, each at
// its own rank.  Runs are cut where a warp's records end.  On the 4096^2
// frame 15.4 M draw records became 4.1 M runs: the row sort went from 0.246
// to 0.107 ms and the resolve from 0.256 to 0.158; in a batch of 64 uneven
// scenes the resolve went from 1.53 to 0.70 ms.
//
// Each thread owns ITEMS consecutive sorted records, whose relations to the
// record before (same cell, same row, cells apart) it keeps as bit masks: the
// runs' starts and ends come from them by a few logic operations for all its
// records at once.  The kernel is bound by instructions and the barriers
// between its phases.  With 64-bit keys, record by record, and starts found
// again from staged keys it issued 257 M warp instructions for 21 M records;
// the split keys, the masks and the paint and row staged with a start leave
// 143 M: with the reduce 0.465 -> 0.281 ms on the 4096^2 frame, 0.30 -> 0.20
// in the batch.  48 registers (a few spilled) for 5 CTAs an SM: 0.301 with 64
// and 4, the same with 40 and 6.
template <int ITEMS, int THREADS> struct RunSmem {
    uint32_t tile;
    int32_t warpA[THREADS / 32];
    int32_t warpAf[THREADS / 32];
    uint32_t warpB[THREADS / 32];                   // starts << 16 | ends of a warp, then of those before
    uint32_t warpC[THREADS / 32];                   // fragments << 16 | spans of a warp
    uint64_t prefixB;
    uint32_t count;
    // per thread: its first record, the centre parts of its leading run (the
    // records of that cell) and whether all its records are in it
    uint32_t run_p[THREADS], run_l[THREADS];
    int32_t run_sum[THREADS];
    uint32_t run_all[THREADS];
    uint32_t next_p, next_l;                        // the record after the tile (path ~0 if none)
    int32_t next_c;                                 // its centre part
    uint32_t start[THREADS * ITEMS];                // j-th start: row in its scene << 16 | first cell
    uint32_t info[THREADS * ITEMS];                 // its paint
    uint32_t row[THREADS * ITEMS];                  // its global row (a batch's)
    uint16_t end[THREADS * ITEMS];                  // j-th end: the cell after the last
};

template <int ITEMS, int THREADS, bool MULTI>
__global__ void __launch_bounds__(THREADS, 5) k_winding_runs(const WindArgs a, const int32_t* __restrict__ tile_in,
                                                             uint64_t* __restrict__ tstat, uint32_t* counter,
                                                             uint32_t* status, uint32_t spin_limit) {
    wait_for_stream();
    constexpr int kTile = THREADS * ITEMS;
    static_assert(ITEMS % 2 == 0 && ITEMS <= 8, "records per thread");
    __shared__ RunSmem<ITEMS, THREADS> S;
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) S.tile = atomicAdd(counter, 1u);
    __syncthreads();
    const uint32_t tile = S.tile;
    const int64_t n = a.n_dev ? (int64_t)min((uint64_t)*a.n_dev, (uint64_t)a.n) : a.n;
    const int64_t tbase = (int64_t)tile * kTile;
    const int64_t num_tiles = (n + kTile - 1) / kTile;
    if (tbase >= n) {
        // launched for the capacity: nothing here
        if (n == 0 && tile == 0 && threadIdx.x == 0 && a.dbg_wscan) a.dbg_wscan[0] = 0;
        return;
    }
    const int32_t t_in = tile_in[tile];
    const KeySplit ks(a.L);
    const uint32_t xbits = a.L.xbits, xmask = (1u << xbits) - 1u, off_rank = (uint32_t)(a.L.Hy - 1);
    const int32_t F = a.F;

    // ---- this thread's records, and the ones before and after them
    const int64_t ibase = tbase + (int64_t)threadIdx.x * ITEMS;
    const int nvalid = (int)max((int64_t)0, min((int64_t)ITEMS, n - ibase));
    uint32_t kp[ITEMS], kl[ITEMS], wbits;
    load_split<ITEMS>(a, ks, ibase, n, kp, kl, wbits, status);
    // the fill rule and paint of the first record's path, fetched early
    uint32_t rule_path = kp[0], paint_path = kp[0], rule = 0, paint = 0;
    if (nvalid > 0) {
        rule = a.fill_rule[rule_path];
        paint = a.fill_info[paint_path];
    }
    uint32_t pprev = __shfl_up_sync(0xFFFFFFFFu, kp[ITEMS - 1], 1), lprev = __shfl_up_sync(0xFFFFFFFFu, kl[ITEMS - 1], 1);
    uint32_t pnext = __shfl_down_sync(0xFFFFFFFFu, kp[0], 1), lnext = __shfl_down_sync(0xFFFFFFFFu, kl[0], 1);
    uint32_t wb = 0;
    if (lane == 0 && ibase > 0 && ibase - 1 < n) split_record(a, ks, ibase - 1, n, pprev, lprev, wb, nullptr);
    wb = 0;
    if (lane == 31 && ibase + ITEMS < n) split_record(a, ks, ibase + ITEMS, n, pnext, lnext, wb, nullptr);
    if (ibase + ITEMS >= n) pnext = ~0u;   // no record after this thread's last
    if (threadIdx.x == THREADS - 1) {
        S.next_p = pnext;
        S.next_l = lnext;
        S.next_c = sx2(wb >> 2);
    }
    // relations to the record before: same cell, same path and row (a key is
    // path, row rank, x + 1), the next cell, a cell further on
    const uint32_t vmask = (1u << nvalid) - 1u;
    uint32_t same = 0, in_row = 0, next_cell = 0;
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const uint32_t p0 = k == 0 ? pprev : kp[k - 1], l0 = k == 0 ? lprev : kl[k - 1];
        const bool sp = p0 == kp[k];
        same |= (sp && l0 == kl[k] ? 1u : 0u) << k;
        in_row |= (sp && (l0 >> xbits) == (kl[k] >> xbits) ? 1u : 0u) << k;
        next_cell |= (l0 + 1u == kl[k] ? 1u : 0u) << k;   // within in_row
    }
    if (ibase == 0) same &= ~1u, in_row &= ~1u;   // record 0 has none before it
    const uint32_t hdm = ~same & vmask;           // first records of a cell

    // ---- winding prefix: the tile's from the tile scan, then the CTA's
    const uint32_t heads = MULTI ? scene_heads<ITEMS>(a, ibase, nvalid, kp, pprev) : 0u;
    bool fe, aggf;
    int32_t ve, agg;
    winding_prefix<THREADS, MULTI>(heads, wbits, S.warpA, S.warpAf, fe, ve, aggf, agg);
    int32_t wrun = fe ? ve : wadd(t_in, ve);

    // ---- centre parts of each record's cell from it to the cell's end
    // (pixel mode): a reverse segmented sum over the records of a cell, with
    // the cell that continues past this thread followed through the others'
    int32_t csum[ITEMS];
    if (a.pixel_mode) {
        const uint32_t pl = kp[ITEMS - 1], ll = kl[ITEMS - 1];
        csum[ITEMS - 1] = sx2(wbits >> (4 * (ITEMS - 1) + 2));
#pragma unroll
        for (int k = ITEMS - 2; k >= 0; --k)
            csum[k] = wadd(sx2(wbits >> (4 * k + 2)), (same >> (k + 1)) & 1u ? csum[k + 1] : 0);
        constexpr uint32_t kInner = ((1u << ITEMS) - 1u) & ~1u;   // records with one of this thread before them
        S.run_p[threadIdx.x] = kp[0];
        S.run_l[threadIdx.x] = kl[0];
        S.run_sum[threadIdx.x] = csum[0];
        S.run_all[threadIdx.x] = nvalid == ITEMS && (same & kInner) == kInner ? 1u : 0u;
        __syncthreads();
        // Only a merged fragment (an on-canvas cell that starts in this
        // thread) needs it; off-canvas records of a path share one key (one
        // per row past its right edge) and are never followed.
        const uint32_t xol = ll & xmask;
        const uint32_t xo_max = (uint32_t)div_F((MULTI ? scene_of_path(a.st, pl).W : a.W) + F - 1, F);
        if (pnext == pl && lnext == ll && nvalid == ITEMS && hdm && (ll >> xbits) != off_rank && xol >= 1u && xol <= xo_max) {
            int32_t tail = 0;
            uint32_t t = threadIdx.x + 1;
            bool follow = true;
            while (follow && t < THREADS) {
                if (S.run_p[t] != pl || S.run_l[t] != ll) {
                    follow = false;
                    break;
                }
                tail = wadd(tail, S.run_sum[t]);
                follow = S.run_all[t] != 0;
                ++t;
            }
            if (follow && S.next_p == pl && S.next_l == ll) {
                tail = wadd(tail, S.next_c);
                // two or more records of the cell past the tile's end (rare)
                for (int64_t j = tbase + kTile + 1; j < n; ++j) {
                    uint32_t p, l, w;
                    split_record(a, ks, j, n, p, l, w, nullptr);
                    if (p != pl || l != ll) break;
                    tail = wadd(tail, sx2(w >> 2));
                }
            }
            // for the records of the last one's cell
            const uint32_t from = 31u - (uint32_t)__clz(hdm);
#pragma unroll
            for (int k = 0; k < ITEMS; ++k)
                if ((uint32_t)k >= from) csum[k] = wadd(csum[k], tail);
        }
    }

    // ---- flags (mark_merged_fragment_and_span.comp:22-93): merged fragments
    // and the spans that end at a record
    uint32_t ffm = 0, sfm = 0;
    // on the canvas: a row of it, and 0 <= x = (xo - 1) F < W, i.e. 1 <= xo <= ceil(W / F)
    const uint32_t xo_max1 = (uint32_t)div_F(a.W + F - 1, F);
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        if (MULTI && ((heads >> k) & 1u)) wrun = 0;
        const int32_t wscan = wrun;
        wrun = wadd(wrun, sx2(wbits >> (4 * k)));
        if ((hdm >> k) & 1u) {
            const uint32_t p1 = kp[k], l1 = kl[k], xo1 = l1 & xmask;
            const uint32_t xo_max = MULTI ? (uint32_t)div_F(scene_of_path(a.st, p1).W + F - 1, F) : xo_max1;
            bool ff = (l1 >> xbits) != off_rank && xo1 >= 1u && xo1 <= xo_max;
            bool sf = ((in_row & ~next_cell) >> k) & 1u;   // cells between the record before and this one
            if (p1 != rule_path) {
                rule = a.fill_rule[p1];
                rule_path = p1;
            }
            sf = sf && rule_pass(rule, wscan);
            // centre sample of the merged cell: scan at its first record plus
            // the left-of-centre changes of the cell's pieces
            if (a.pixel_mode) ff = ff && rule_pass(rule, wadd(wscan, csum[k]));
            ffm |= (ff ? 1u : 0u) << k;
            sfm |= (sf ? 1u : 0u) << k;
            if (a.path_draw && (ff || sf)) atomicAdd(&a.path_draw[p1], (ff ? 1u : 0u) + (sf ? 1u : 0u));
        }
        if (a.dbg_wscan && k < nvalid) {
            const int64_t i = ibase + k;
            a.dbg_wscan[i] = wscan;
            a.dbg_fflag[i] = (int32_t)((ffm >> k) & 1u);
            a.dbg_sflag[i] = (int32_t)((sfm >> k) & 1u);
            a.dbg_skey[i] = unpack_key(a.L, ((uint64_t)kp[k] << ks.pshift) | kl[k]).yx;
        }
    }

    // ---- runs: is the cell before each record painted?  Before this thread's
    // first head, that of the last head of a lane before, of this warp.
    const uint32_t hm = __ballot_sync(0xFFFFFFFFu, hdm != 0);
    const uint32_t pm = __ballot_sync(0xFFFFFFFFu, hdm != 0 && ((ffm >> (31 - __clz(hdm | 1u))) & 1u));
    const uint32_t vm = __ballot_sync(0xFFFFFFFFu, nvalid > 0);
    const uint32_t below = hm & lanemask_lt();
    uint32_t painted = below ? (pm >> (31 - __clz(below))) & 1u : 0u, pmask = 0;
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        pmask |= painted << k;
        painted = (hdm >> k) & 1u ? (ffm >> k) & 1u : painted;
    }
    const uint32_t joined = pmask & in_row & (sfm | (ffm & next_cell));
    const uint32_t ends_prev = hdm & pmask & ~joined;    // the cell before was the last of a run
    const uint32_t starts = (sfm | ffm) & ~joined;       // with the span before the record, or with its cell
    const uint32_t ends_span = sfm & ~ffm;               // the span before the record was
    // the warp's last records: a run does not go on into the next warp
    const bool ends_warp = painted && vm && lane == 31u - (uint32_t)__clz(vm);
    const uint32_t drawn = __reduce_add_sync(0xFFFFFFFFu, ((uint32_t)__popc(ffm) << 16) | (uint32_t)__popc(sfm));
    if (lane == 0) S.warpC[warp] = drawn;

    // ---- output slots: starts and ends packed 16:16 within the CTA (as many
    // of the one as of the other), runs across tiles with a look-back
    const uint32_t bsum =
        ((uint32_t)__popc(starts) << 16) | (uint32_t)(__popc(ends_prev) + __popc(ends_span) + (ends_warp ? 1 : 0));
    const uint32_t inclB = warp_incl<uint32_t>(bsum);
    if (lane == 31) S.warpB[warp] = inclB;
    __syncthreads();
    if (warp == 0) {
        const uint32_t w = lane < THREADS / 32 ? S.warpB[lane] : 0u;
        const uint32_t wi = warp_incl<uint32_t>(w);
        if (lane < THREADS / 32) S.warpB[lane] = wi - w;
        const uint32_t runs = __shfl_sync(0xFFFFFFFFu, wi, THREADS / 32 - 1) >> 16;
        if (lane == 0) st_relaxed_u64(&tstat[tile], (tile == 0 ? kFlagP : kFlagA) | runs);
        const uint32_t d = __reduce_add_sync(0xFFFFFFFFu, lane < THREADS / 32 ? S.warpC[lane] : 0u);
        if (lane < 2) {
            const uint32_t v = lane ? d & 0xFFFFu : d >> 16;
            if (v) atomicAdd(reinterpret_cast<unsigned long long*>(&a.totals[lane]), (unsigned long long)v);
        }
        uint64_t excl = 0;
        if (tile > 0) {
            excl = lookback(tstat, tile, status, spin_limit);
            if (lane == 0) st_relaxed_u64(&tstat[tile], kFlagP | (excl + runs));
        }
        if (lane == 0) {
            S.prefixB = excl;
            S.count = runs;
            if (tile == num_tiles - 1) *a.n_draw = (uint32_t)(excl + runs);
        }
    }
    __syncthreads();
    // this thread's starts and ends at their ranks.  Cells are x - 1: the cell
    // after that of the record before is its x, the one before this record's
    // is x - 2.  A painted record is on the canvas: rank Hy is row 0, rank
    // r < Hy - 1 is row r + 1.
    {
        const uint32_t l0 = S.warpB[warp] + (inclB - bsum);
        uint32_t rs = l0 >> 16, re = l0 & 0xFFFFu;
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            const uint32_t x0 = (k == 0 ? lprev : kl[k - 1]) & xmask, x1 = kl[k] & xmask;
            if ((ends_prev >> k) & 1u) S.end[re++] = (uint16_t)x0;
            if ((ends_span >> k) & 1u) S.end[re++] = (uint16_t)(x1 - 1u);
            if ((starts >> k) & 1u) {
                const uint32_t p1 = kp[k], rank = kl[k] >> xbits;
                const uint32_t yy = rank == (uint32_t)a.L.Hy ? 0u : rank + 1u;
                if (p1 != paint_path) {
                    paint = a.fill_info[p1];
                    paint_path = p1;
                }
                S.start[rs] = (yy << 16) | ((sfm >> k) & 1u ? x0 : x1 - 1u);
                S.info[rs] = paint;
                if (MULTI) S.row[rs] = scene_of_path(a.st, p1).row_base + yy;
                ++rs;
            }
        }
        if (ends_warp) {
            // the last record's cell, which is that of the last head
            uint32_t x = lprev;
#pragma unroll
            for (int k = 0; k < ITEMS; ++k) x = (hdm >> k) & 1u ? kl[k] : x;
            S.end[re] = (uint16_t)(x & xmask);
        }
    }
    __syncthreads();

    // ---- the runs, one a thread.  Each also adds to its row's run count and
    // pixel sum (summed over the lanes of a warp that share the row), and an
    // opaque one to the cuts of the resolve segments it covers whole.  Every
    // lane of a warp runs the same rounds (the row sums are warp-wide).
    const int64_t tile_first = (int64_t)S.prefixB;
    const uint32_t tile_cnt = S.count;
    const uint32_t rounds_end = (tile_cnt + THREADS - 1) / THREADS * THREADS;
    for (uint32_t j = threadIdx.x; j < rounds_end; j += THREADS) {
        uint32_t row = 0xFFFFFFFFu, px = 0;
        bool counted = false;
        if (j < tile_cnt) {
            const uint32_t st = S.start[j], info = S.info[j];
            row = MULTI ? S.row[j] : st >> 16;
            const int32_t x0 = (int32_t)(st & 0xFFFFu) * F, x1 = (int32_t)S.end[j] * F, y = (int32_t)(st >> 16) * F;
            const int64_t o = tile_first + j;
            // only runs inside the capacity are written and counted, so that
            // the row sort and the resolve stay inside the buffers
            if (o < a.draw_capacity) {
                a.draw[o] = make_int4((int32_t)((uint32_t)y << 16) | x0, x1 - x0, (int32_t)info, 0);
                a.draw_row[o] = row;
                px = (uint32_t)imax(x1 - x0, 0);
                counted = row < a.cut_rows;
                // a run that hides everything under it ends the resolve's work
                // before it in each segment it covers whole
                if (counted && a.pixel_mode && (info >> 24) == 255u) {
                    const int32_t s_hi = imin(x1 / kResolveSeg, (int32_t)a.cut_segs);
                    for (int32_t sg = (x0 + kResolveSeg - 1) / kResolveSeg; sg < s_hi; ++sg)
                        atomicMax(&a.seg_cut[(size_t)row * a.cut_segs + (uint32_t)sg], (uint32_t)o + 1u);
                }
            } else {
                set_error(status, ERR_CAPACITY);
            }
        }
        const uint32_t peers = __match_any_sync(0xFFFFFFFFu, counted ? row : 0xFFFFFFFFu);
        if (counted) {
            const uint32_t cnt = __popc(peers);
            const uint32_t psum = __reduce_add_sync(peers, px);
            if (lane == (uint32_t)(__ffs(peers) - 1)) {
                atomicAdd(&a.row_count[row], cnt);
                atomicAdd(&a.row_px[row], (unsigned long long)psum);
            }
        }
    }
}
// Tiles of 256 threads with 4 or 8 records each.
static int64_t wind_tile(int items) { return items == 4 ? 1024 : 2048; }

size_t winding_status_words(int64_t n, int items) {
    const int64_t tile = wind_tile(items);
    return (size_t)((n + tile - 1) / tile + 1);
}
// tile pairs (64-bit), then tile prefixes (32-bit)
size_t winding_tile_words(int64_t n, int items) { return 2 * winding_status_words(n, items); }

// Tiles from which a warp reduces one: 8 warps of a CTA on each of 152 SMs.
constexpr int64_t kWarpTiles = 4 * 8 * 152;

template <int ITEMS, bool MULTI>
static void launch_runs(const WindArgs& a, int64_t tiles, uint64_t* words, uint64_t* tagg, int32_t* tile_in,
                        uint32_t* counters, uint32_t* status, cudaStream_t st) {
    if (tiles >= kWarpTiles)
        launch_after(k_winding_reduce<ITEMS, 256, 1, MULTI>, (unsigned)((tiles + 7) / 8), 256, 0, st, a, tagg, tile_in,
                     counters + 1);
    else
        launch_after(k_winding_reduce<ITEMS, 256, 8, MULTI>, (unsigned)tiles, 256, 0, st, a, tagg, tile_in,
                     counters + 1);
    launch_after(k_winding_runs<ITEMS, 256, MULTI>, (unsigned)tiles, 256, 0, st, a, tile_in, words, counters, status,
                 spin_limit());
}

void launch_winding_emit(const WindArgs& a, int items, uint64_t* tile_status, uint64_t* tile_sums, uint32_t* counters,
                         uint32_t* status, cudaStream_t st) {
    if (a.n <= 0) return;
    const int64_t tile = wind_tile(items);
    const int64_t tiles = (a.n + tile - 1) / tile;
    int32_t* tile_in = reinterpret_cast<int32_t*>(tile_sums + (tiles + 1));
    count_launches(2);
    const bool multi = a.st.n_scenes > 1;
    if (items == 4)
        (multi ? launch_runs<4, true> : launch_runs<4, false>)(a, tiles, tile_status, tile_sums, tile_in, counters,
                                                               status, st);
    else
        (multi ? launch_runs<8, true> : launch_runs<8, false>)(a, tiles, tile_status, tile_sums, tile_in, counters,
                                                               status, st);
}

void launch_draw_list(const WindArgs& a, int items, uint64_t* tile_status, const uint64_t* tile_sums,
                      uint32_t* counters, uint32_t* status, cudaStream_t st) {
    if (a.n <= 0) return;
    const int64_t tile = wind_tile(items);
    const int64_t tiles = (a.n + tile - 1) / tile;
    const int32_t* tile_in = reinterpret_cast<const int32_t*>(tile_sums + (tiles + 1));
    count_launches(1);
    if (items == 4)
        k_draw_list<4, 256><<<(unsigned)tiles, 256, 0, st>>>(a, tile_in, tile_status, counters, status,
                                                                            spin_limit());
    else
        k_draw_list<8, 256><<<(unsigned)tiles, 256, 0, st>>>(a, tile_in, tile_status, counters, status,
                                                                            spin_limit());
}

}  // namespace sr
