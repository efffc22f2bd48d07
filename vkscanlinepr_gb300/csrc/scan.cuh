// scan.cuh — the tile of a single-pass exclusive scan (decoupled look-back),
// shared by the standalone scan and the kernels that scan as part of their
// work.
//
// A tile publishes its aggregate, then one warp looks back over its
// predecessors' words.  A word carries its flag and its value together, so
// relaxed accesses suffice: nothing else is read on its authority.  Every
// spin is bounded: after the spin limit's polls the tile records
// ERR_LOOKBACK_TIMEOUT and carries on, so a stalled predecessor can never
// hang the GPU.
#pragma once
#include "common.cuh"

namespace sr {

constexpr uint64_t kScanFlagA = 1ull << 62;   // aggregate of the tile
constexpr uint64_t kScanFlagP = 2ull << 62;   // sum up to and including it

SR_DEV uint64_t ld_relaxed_u64(const uint64_t* p) {
    uint64_t v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
SR_DEV void st_relaxed_u64(uint64_t* p, uint64_t v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

SR_DEV int32_t warp_incl_scan(int32_t v) {
    const uint32_t lane = lane_id();
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int32_t t = __shfl_up_sync(0xFFFFFFFFu, v, d);
        if ((int)lane >= d) v = wadd(v, t);
    }
    return v;
}

// Warp-cooperative look-back over 64-bit tile words (flag in bits 62-63,
// value in bits 0-31).  Returns the sum of all predecessors of `tile`.  (Steps
// over four windows of 32 words were slower: the polls of the CTAs that wait
// slow each other down.)
SR_DEV int32_t lookback_i32(uint64_t* tstat, uint32_t tile, uint32_t* status, uint32_t spin_limit) {
    const uint32_t lane = lane_id();
    int32_t excl = 0;
    int64_t look = (int64_t)tile - 1;
    uint32_t spins = 0;
    while (look >= 0) {
        const int64_t j = look - (int64_t)lane;
        const uint64_t s = j >= 0 ? ld_relaxed_u64(&tstat[j]) : kScanFlagP;
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
        const int32_t v = ((int)lane <= firstp) ? (int32_t)(uint32_t)s : 0;
        excl = wadd(excl, (int32_t)__reduce_add_sync(0xFFFFFFFFu, (uint32_t)v));
        if (pm) break;
        look -= 32;
    }
    return excl;
}

// Exclusive prefix of one value per thread over all tiles (tile ids from a
// counter, so every predecessor is running or done): the CTA's own scan, then
// the look-back.  s_warp: THREADS / 32 + 1 words.  Every thread gets its
// prefix; *tile_total, the sum up to and including this tile.  tstat NULL: the
// only tile, starting from `carry`.
template <int THREADS>
SR_DEV int32_t scan_thread_values(int32_t v, uint32_t tile, uint64_t* tstat, uint32_t* status, uint32_t spin_limit,
                                  int32_t* s_warp, int32_t* tile_total, int32_t carry = 0) {
    constexpr int kWarps = THREADS / 32;
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    const int32_t incl = warp_incl_scan(v);
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        const int32_t w = lane < kWarps ? s_warp[lane] : 0;
        const int32_t wi = warp_incl_scan(w);
        const int32_t agg = __shfl_sync(0xFFFFFFFFu, wi, kWarps - 1);
        if (tstat && lane == 0) st_relaxed_u64(&tstat[tile], (tile == 0 ? kScanFlagP : kScanFlagA) | (uint32_t)agg);
        int32_t excl = carry;
        if (tile > 0) {
            excl = lookback_i32(tstat, tile, status, spin_limit);
            if (lane == 0) st_relaxed_u64(&tstat[tile], kScanFlagP | (uint32_t)wadd(excl, agg));
        }
        if (lane < kWarps) s_warp[lane] = wadd(excl, wadd(wi, -w));
        if (lane == 0) s_warp[kWarps] = wadd(excl, agg);
    }
    __syncthreads();
    *tile_total = s_warp[kWarps];
    return wadd(s_warp[warp], wadd(incl, -v));
}

// The tile's values in registers (row r of a warp: 128 consecutive values,
// four neighbouring ones a lane), scanned into out.  Returns true in the tile
// that holds the end (it has written out[n]).
template <int ROWS, int THREADS>
SR_DEV bool scan_tile_values(const int4 (&v)[ROWS], int32_t* out, int64_t n, uint32_t tile, uint64_t* tstat,
                             uint32_t* status, uint32_t spin_limit, int32_t* s_warp, int32_t* total,
                             int32_t carry = 0) {
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    const int64_t base = ((int64_t)tile * (THREADS / 32) + warp) * (128 * ROWS) + lane * 4;
    const bool out4 = (reinterpret_cast<uintptr_t>(out) & 15) == 0;
    // the lane's prefix in each row, and the warp's sum
    int32_t ex[ROWS];
    int32_t run = 0;
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        const int32_t s = wadd(wadd(v[r].x, v[r].y), wadd(v[r].z, v[r].w));
        const int32_t incl = warp_incl_scan(s);
        ex[r] = wadd(run, wadd(incl, -s));
        run = wadd(run, __shfl_sync(0xFFFFFFFFu, incl, 31));
    }
    // the warps' sums: lane 0 brings its warp's into the CTA's scan, whose
    // value for lane 0 is what comes before the warp
    int32_t before = scan_thread_values<THREADS>(lane == 0 ? run : 0, tile, tstat, status, spin_limit, s_warp, total, carry);
    before = __shfl_sync(0xFFFFFFFFu, before, 0);
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        const int64_t i = base + r * 128;
        int4 q;
        q.x = wadd(before, ex[r]);
        q.y = wadd(q.x, v[r].x);
        q.z = wadd(q.y, v[r].y);
        q.w = wadd(q.z, v[r].z);
        if (out4 && i + 4 <= n) {
            *reinterpret_cast<int4*>(out + i) = q;
        } else {
            if (i < n) out[i] = q.x;
            if (i + 1 < n) out[i + 1] = q.y;
            if (i + 2 < n) out[i + 2] = q.z;
            if (i + 3 < n) out[i + 3] = q.w;
        }
    }
    const bool last = (int64_t)(tile + 1) * (THREADS * 4 * ROWS) >= n;
    if (last && threadIdx.x == 0) out[n] = *total;
    return last;
}

// The tile's values from memory: whole lines, zeros past n.
template <int ROWS, int THREADS>
SR_DEV void load_tile_values(int4 (&v)[ROWS], const int32_t* in, int64_t n, uint32_t tile) {
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    const int64_t base = ((int64_t)tile * (THREADS / 32) + warp) * (128 * ROWS) + lane * 4;
    const bool in4 = (reinterpret_cast<uintptr_t>(in) & 15) == 0;
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        const int64_t i = base + r * 128;
        if (in4 && i + 4 <= n) {
            v[r] = *reinterpret_cast<const int4*>(in + i);
        } else {
            v[r].x = i < n ? in[i] : 0;
            v[r].y = i + 1 < n ? in[i + 1] : 0;
            v[r].z = i + 2 < n ? in[i + 2] : 0;
            v[r].w = i + 3 < n ? in[i + 3] : 0;
        }
    }
}

// One tile of the exclusive scan of in[0, n) into out[0, n]: THREADS x 4 x
// ROWS values.  Returns true in the tile that holds the end.  in and out may
// alias.
template <int ROWS, int THREADS>
SR_DEV bool scan_tile_i32(const int32_t* in, int32_t* out, int64_t n, uint32_t tile, uint64_t* tstat,
                          uint32_t* status, uint32_t spin_limit, int32_t* s_warp, int32_t* total, int32_t carry = 0) {
    int4 v[ROWS];
    load_tile_values<ROWS, THREADS>(v, in, n, tile);
    return scan_tile_values<ROWS, THREADS>(v, out, n, tile, tstat, status, spin_limit, s_warp, total, carry);
}

}  // namespace sr
