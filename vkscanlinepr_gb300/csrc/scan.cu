// scan.cu — the standalone exclusive scan.
//
// Replaces naive_scan.comp:27-73, which runs in ONE workgroup and walks the
// input in dependent batches of 1023.  Output: out[0..n], out[n] = total
// (exactly n+1 writes).
//   * Short inputs: one CTA, one launch, no scratch.
//   * Longer ones: every CTA sums a chunk, then every CTA adds up the sums
//     before its chunk and scans it.  The input is read twice (a part of it
//     from the L2), but nothing waits for anything within a launch: 50 M
//     values take 98 us (400 MB of input and output at 4.1 TB/s), 1 M take
//     10.8, where a single pass took 151 and 15, its look-back moving on 32
//     tiles a memory round trip whatever the tiles' size (16,384-value tiles
//     119; persistent CTAs with their loads running ahead 189).
//   * k_scan_i32 is the single pass with decoupled look-back that the frame's
//     own scans use (scan.cuh); here it only serves the check of its bounded
//     wait.
#include <algorithm>

#include "kernels.h"
#include "scan.cuh"

namespace sr {

namespace {
constexpr int kThreads = 256, kRows = 4, kTile = kThreads * 4 * kRows;
// Up to kOneTo values one CTA scans all, in rounds, without scratch: 10,007
// values take 4.2 us where the chunks take 8.7 (the single-pass scan with its
// allocation and clear took 9.5), 32,768 take 7.8 and 8.5.
constexpr int kOneThreads = 1024, kOneRows = 4, kOneTile = kOneThreads * 4 * kOneRows;
constexpr int64_t kOneTo = 32768;
// Above, at most kChunksMax chunks of whole tiles: four CTAs an SM (three, or
// two of 512 threads: the same within 1%).
constexpr int kChunkCtas = 4;
constexpr uint32_t kChunksMax = 152 * kChunkCtas;

// Tiles [t0, t1) of chunk c.
SR_DEV void chunk_tiles(uint32_t tiles, uint32_t& t0, uint32_t& t1) {
    const uint32_t per = tiles / gridDim.x, more = tiles % gridDim.x, c = blockIdx.x;
    t0 = c * per + min(c, more);
    t1 = t0 + per + (c < more ? 1u : 0u);
}

SR_DEV int32_t cta_sum(int32_t v, int32_t* s_warp) {
    v = (int32_t)__reduce_add_sync(0xFFFFFFFFu, (uint32_t)v);
    if (lane_id() == 0) s_warp[threadIdx.x >> 5] = v;
    __syncthreads();
    int32_t t = 0;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) t = wadd(t, s_warp[w]);
    return t;
}
}  // namespace

__global__ void __launch_bounds__(kThreads) k_scan_i32(const int32_t* in, int32_t* out, int64_t n, uint64_t* tstat,
                                                       uint32_t* counter, uint32_t* status, uint32_t spin_limit) {
    __shared__ uint32_t s_tile;
    __shared__ int32_t s_warp[kThreads / 32 + 1];
    if (threadIdx.x == 0) s_tile = atomicAdd(counter, 1u);
    __syncthreads();
    int32_t total;
    scan_tile_i32<kRows, kThreads>(in, out, n, s_tile, tstat, status, spin_limit, s_warp, &total);
}

__global__ void __launch_bounds__(kOneThreads) k_scan_one(const int32_t* in, int32_t* out, int64_t n) {
    wait_for_stream();
    __shared__ int32_t s_warp[2][kOneThreads / 32 + 1];
    int32_t carry = 0;
    int par = 0;
    for (int64_t base = 0; base < n; base += kOneTile, par ^= 1) {
        int32_t total;
        scan_tile_i32<kOneRows, kOneThreads>(in + base, out + base, n - base, 0u, nullptr, nullptr, 0u, s_warp[par],
                                             &total, carry);
        carry = total;
    }
}

// Sum of each chunk, read from its end back, so that what the scan reads
// first is what the L2 holds.
__global__ void __launch_bounds__(kThreads, 8) k_chunk_sums(const int32_t* __restrict__ in, int64_t n, uint32_t tiles,
                                                            int32_t* __restrict__ sums) {
    wait_for_stream();
    __shared__ int32_t s_warp[kThreads / 32];
    uint32_t t0, t1;
    chunk_tiles(tiles, t0, t1);
    int32_t v = 0;
#pragma unroll 2
    for (uint32_t t = t1; t > t0; --t) {
        int4 q[kRows];
        load_tile_values<kRows, kThreads>(q, in, n, t - 1);
#pragma unroll
        for (int r = 0; r < kRows; ++r) v = wadd(v, wadd(wadd(q[r].x, q[r].y), wadd(q[r].z, q[r].w)));
    }
    v = cta_sum(v, s_warp);
    if (threadIdx.x == 0) sums[blockIdx.x] = v;
}

// The chunks' scans, the next tile's loads under way while one is scanned.
__global__ void __launch_bounds__(kThreads, kChunkCtas) k_chunk_scan(const int32_t* in, int32_t* out, int64_t n,
                                                                     uint32_t tiles, const int32_t* __restrict__ sums) {
    wait_for_stream();
    __shared__ int32_t s_warp[2][kThreads / 32 + 1];
    uint32_t t0, t1;
    chunk_tiles(tiles, t0, t1);
    int4 next[kRows];
    load_tile_values<kRows, kThreads>(next, in, n, t0);
    int32_t before = 0;
    for (uint32_t c = threadIdx.x; c < blockIdx.x; c += kThreads) before = wadd(before, sums[c]);
    int32_t carry = cta_sum(before, s_warp[1]);
    int par = 0;
    for (uint32_t t = t0; t < t1; ++t, par ^= 1) {
        int4 v[kRows];
#pragma unroll
        for (int r = 0; r < kRows; ++r) v[r] = next[r];
        if (t + 1 < t1) load_tile_values<kRows, kThreads>(next, in, n, t + 1);
        int32_t total;
        const int64_t first = (int64_t)t * kTile;
        scan_tile_values<kRows, kThreads>(v, out + first, n - first, 0u, nullptr, nullptr, 0u, s_warp[par], &total,
                                          carry);
        carry = total;
    }
}

// Sticky error bits of the standalone scans on each device that loads the
// library (4 bytes, held until exit).
static __device__ uint32_t g_standalone_scan_status;

cudaError_t standalone_scan_status(uint32_t** out) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_standalone_scan_status);
    *out = static_cast<uint32_t*>(p);
    return e;
}

static uint32_t tiles_of(int64_t n) { return (uint32_t)((n + kTile - 1) / kTile); }

size_t scan_scratch_bytes(int64_t n) { return n <= kOneTo ? 0 : sizeof(int32_t) * std::min(tiles_of(n), kChunksMax); }

void launch_scan_i32(const int32_t* in, int32_t* out, int64_t n, void* scratch, cudaStream_t st) {
    if (n <= 0) {
        cudaMemsetAsync(out, 0, sizeof(int32_t), st);
        return;
    }
    if (n <= kOneTo) {
        count_launches(1);
        launch_after(k_scan_one, 1, kOneThreads, 0, st, in, out, n);
        return;
    }
    count_launches(2);
    const uint32_t tiles = tiles_of(n);
    const unsigned grid = std::min(tiles, kChunksMax);
    launch_after(k_chunk_sums, grid, kThreads, 0, st, in, n, tiles, static_cast<int32_t*>(scratch));
    launch_after(k_chunk_scan, grid, kThreads, 0, st, in, out, n, tiles, static_cast<const int32_t*>(scratch));
}

size_t lookback_scan_words(int64_t n) { return (size_t)tiles_of(n) + 1; }

void launch_lookback_scan_i32(const int32_t* in, int32_t* out, int64_t n, uint64_t* tile_status,
                              uint32_t* tile_counter, uint32_t* status, cudaStream_t st) {
    count_launches(1);
    k_scan_i32<<<tiles_of(n), kThreads, 0, st>>>(in, out, n, tile_status, tile_counter, status, spin_limit());
}

}  // namespace sr
