// noalloc.cu — the exclusive scan for callers that cannot allocate device
// memory.
//
// sr_exclusive_scan_i32 takes its scratch from a memory pool.
// Some callers cannot allow that: a host that hands all device memory to
// its own allocator or runs under a hard memory budget forbids third-party
// allocations, and a frame loop with a fixed latency budget cannot risk an
// allocation call that may wait on the device.  This variant launches the same
// kernels with their scratch in a fixed array compiled into the library: every
// GPU that loads the library holds SR_NOALLOC_SCAN_SCRATCH_BYTES of it until
// the process exits.
#include <cstdarg>
#include <cstdio>
#include <mutex>

#include "../../include/sr.h"
#include "kernels.h"

namespace sr {
sr_status report_error(sr_status s, const char* msg);   // api.cu
}

namespace {

// More than any scan's scratch (scan_scratch_bytes).
constexpr size_t kNoallocWords = SR_NOALLOC_SCAN_SCRATCH_BYTES / sizeof(uint64_t);

static __device__ __align__(256) uint64_t g_noalloc_scan_scratch[kNoallocWords];

constexpr int kMaxDevices = 64;
std::mutex g_mutex;
uint64_t* g_scratch_addr[kMaxDevices] = {};

// Device address, on the current device, of the scratch array, looked up once
// per device (the array's name in host code is only a stand-in).  A
// cudaDeviceReset unloads the library's device code, so it does not survive
// one.
sr_status scratch_on_current_device(uint64_t** scratch) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return sr::report_error(SR_ERR_CUDA, cudaGetErrorString(e));
    if (dev < 0 || dev >= kMaxDevices) return sr::report_error(SR_ERR_INVALID_ARG, "device ordinal above 63");
    std::lock_guard<std::mutex> lock(g_mutex);
    if (!g_scratch_addr[dev]) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_scan_scratch);
        if (e != cudaSuccess || !p) return sr::report_error(SR_ERR_CUDA, cudaGetErrorString(e));
        g_scratch_addr[dev] = static_cast<uint64_t*>(p);
    }
    *scratch = g_scratch_addr[dev];
    return SR_OK;
}

}  // namespace

extern "C" sr_status sr_exclusive_scan_i32_noalloc(const int32_t* d_in, int32_t* d_out, int64_t n, void* stream) {
    if (n < 0 || n > SR_NOALLOC_SCAN_MAX_N) {
        char msg[160];
        snprintf(msg, sizeof msg, "scan length %lld outside 0..%lld (the fixed scratch of the allocation-free scan)",
                 (long long)n, (long long)SR_NOALLOC_SCAN_MAX_N);
        return sr::report_error(SR_ERR_INVALID_ARG, msg);
    }
    if (!d_out || (n > 0 && !d_in)) return sr::report_error(SR_ERR_INVALID_ARG, "NULL device pointer");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    uint64_t* scratch = nullptr;
    sr_status s = scratch_on_current_device(&scratch);
    if (s != SR_OK) return s;
    // the sums of the previous call stay in the array; a scan writes what it
    // reads of it
    if (sr::scan_scratch_bytes(n) > sizeof(uint64_t) * kNoallocWords)
        return sr::report_error(SR_ERR_INTERNAL, "scan scratch too small");
    sr::launch_scan_i32(d_in, d_out, n, scratch, st);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? SR_OK : sr::report_error(SR_ERR_CUDA, cudaGetErrorString(e));
}
