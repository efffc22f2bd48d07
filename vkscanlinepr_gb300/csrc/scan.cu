// scan.cu — the standalone exclusive scan.
//
// Replaces naive_scan.comp:27-73, which runs in ONE workgroup and walks the
// input in dependent batches of 1023.  Here every CTA scans a tile and looks
// back over its predecessors' published sums (scan.cuh).  Output:
// out[0..n], out[n] = total (exactly n+1 writes).
#include "kernels.h"
#include "scan.cuh"

namespace sr {

namespace {
constexpr int kThreads = 256;
constexpr int kRows = 4;
constexpr int kTile = kThreads * 4 * kRows;
}  // namespace

__global__ void __launch_bounds__(kThreads) k_scan_i32(const int32_t* in, int32_t* out, int64_t n,
                                                       uint64_t* tstat, uint32_t* counter, uint32_t* status,
                                                       uint32_t spin_limit) {
    __shared__ uint32_t s_tile;
    __shared__ int32_t s_warp[kThreads / 32 + 1];
    if (threadIdx.x == 0) s_tile = atomicAdd(counter, 1u);
    __syncthreads();
    int32_t total;
    scan_tile_i32<kRows, kThreads>(in, out, n, s_tile, tstat, status, spin_limit, s_warp, &total);
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

size_t scan_status_words(int64_t n) { return (size_t)((n + kTile - 1) / kTile + 1); }

void launch_exclusive_scan_i32(const int32_t* in, int32_t* out, int64_t n, uint64_t* tile_status,
                               uint32_t* tile_counter, uint32_t* status, cudaStream_t st) {
    if (n <= 0) {
        cudaMemsetAsync(out, 0, sizeof(int32_t), st);
        return;
    }
    int64_t tiles = (n + kTile - 1) / kTile;
    count_launches(1);
    k_scan_i32<<<(unsigned)tiles, kThreads, 0, st>>>(in, out, n, tile_status, tile_counter, status, spin_limit());
}

}  // namespace sr
