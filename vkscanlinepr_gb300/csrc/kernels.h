// kernels.h — launch interface between the host orchestration and the
// device kernels of the scanline renderer.
#pragma once
#include <atomic>
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "common.cuh"

namespace sr {

// Number of kernels this library has launched in this process.
void count_launches(uint32_t n);
// Runs fn (setting a kernel attribute) unless it has already run for
// `flags` on the current device (one bit per device, up to 32 devices).
// The bit is set after fn, so no thread skips it before it has taken
// effect; two threads may both run it, which is harmless.
template <typename Fn> void once_per_device(std::atomic<uint32_t>& flags, Fn&& fn) {
    int dev = 0;
    cudaGetDevice(&dev);
    const uint32_t bit = 1u << (dev & 31);
    if (flags.load(std::memory_order_acquire) & bit) return;
    fn();
    flags.fetch_or(bit, std::memory_order_release);
}
uint64_t launches_so_far();
// Launches kernel k (which begins with wait_for_stream()) behind the work in
// st: its CTAs may be placed while the kernel before it drains, so the gap
// between two kernels of a frame is not the launch of the second (a 1024^2
// frame of 14 kernels: 212 -> 186 us; a scan of 10,007 values: 4.1 -> 2.6).
template <class... P, class... A>
void launch_after(void (*k)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t st, const A&... a) {
    cudaLaunchAttribute early{};
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(grid);
    c.blockDim = dim3(block);
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = &early;
    c.numAttrs = 1;
    cudaLaunchKernelEx(&c, k, static_cast<P>(a)...);
}
// Polls a bounded device spin makes before it gives up: kSpinLimitDefault
// unless sr_set_spin_limit chose another.  Read at each launch.
uint32_t spin_limit();
// Device address, on the current device, of the sticky error word of the
// standalone scans (sr_exclusive_scan_i32 and its allocation-free variant),
// which sr_scan_status reads and clears.
cudaError_t standalone_scan_status(uint32_t** out);

struct Mvp {
    float m[16];   // rows m0..m3
};

// One scene of a batch (device layout).  Paths of scene s are
// [path_begin, path_end) in the batch's global path order; its cell rows
// are [row_base, row_base + rows) of the batch's global row order; its
// framebuffer starts at pixel image_off.
struct SceneInfo {
    int32_t W, H;
    uint32_t path_begin, path_end;
    uint32_t row_base, rows;
    uint64_t image_off;
    float mvp[16];
};

struct SceneTable {
    const SceneInfo* scenes;
    const uint32_t* path_scene;   // [n_paths] scene of each path
    uint32_t n_scenes;
};

SR_DEV const SceneInfo& scene_of_path(const SceneTable& t, uint32_t path) { return t.scenes[t.path_scene[path]]; }

// Scene + per-frame arrays the geometry kernels read.  W and H are the
// largest canvas of the batch (key layout); each scene's own canvas comes
// from the scene table.
struct GeomArgs {
    uint32_t n_curves, n_paths;
    const uint32_t* curve_type;
    const uint32_t* curve_pos;
    const uint32_t* curve_path;
    const float2* tpos;
    const int32_t* path_visible;
    float2* curve_end;   // [n_curves] each curve's point at t = 1 (written by the count pass)
    uint32_t* path_begin;   // [n_paths + 1] first curve of each path (likewise)
    int32_t W, H, F;
    int32_t pixel_mode;
    KeyLayout L;
    SceneTable st;
    int64_t rec_cap;   // capacity of the record buffers; larger counts are an overflow
};

// Optional reference-layout outputs for parity dumps (all NULL in production).
struct DebugOut {
    int32_t* fkey;      // [N] packed yx
    int32_t* fwn;       // [N] winding change
    int32_t* fleft;     // [N] centre-sample part (pixel mode)
};

// Crossing-chain work of the intersection stage.
struct ChainWork {
    uint4* pieces;            // [n_curves][5] per-piece chain set-up
    uint32_t* chain_items;    // [list_cap] (curve << 4 | piece << 1 | side), append order
    uint8_t* chain_keys;      // [list_cap] class of each: length class / type
    uint32_t* sorted_items;   // [list_cap] the same, longest class first
    uint4* chain_piece;       // [list_cap] each sorted item's piece, for the record order
    uint32_t list_cap;
    uint32_t* chain_count;    // [1] zeroed before the count pass, as are the next three
    uint32_t* class_count;    // [kChainClassWords] chains of each class
    uint32_t* class_next;     // [kChainClassWords] next place of each class in sorted_items
    uint32_t* chain_queue;    // [1] next ticket of the chains
};
constexpr int kChainClassWords = 64;
// A frame has fewer records (its offsets and counts are 32-bit).
constexpr uint32_t kMaxRecords = 1u << 30;
size_t piece_table_bytes(uint32_t n_curves);
uint32_t chain_list_capacity(uint32_t n_curves);

// Arcs' control and weight slots after launch_transform (SR_CURVE_ARC).
void launch_arc_fixup(const uint32_t* curve_type, const uint32_t* curve_pos, const uint32_t* curve_path,
                      uint32_t n_curves, const float2* pos, const SceneTable& t, float2* tpos, int32_t* path_visible,
                      cudaStream_t st);
// zero: zero_bytes (a multiple of 16) to clear beside it.
void launch_transform(const float2* pos, const uint32_t* pos_path, uint32_t n_points, const SceneTable& t,
                      float2* tpos, int32_t* path_visible, void* zero, size_t zero_bytes, int sm_count, cudaStream_t st);
void launch_count(const GeomArgs& g, float* cut_cache, int32_t* count, const ChainWork& w, uint32_t* status,
                  cudaStream_t st);
// After the count pass: the curves' record offsets offs[0..C] (exclusive scan
// of count, look-back words and counter zeroed; the total also to report_n; a
// capacity error from kMaxRecords on) and the chains in class order.
size_t offset_scan_words(uint32_t n_curves);
void launch_offsets_and_order(const GeomArgs& g, const int32_t* count, int32_t* offs, const ChainWork& w,
                              uint64_t* tile_status, uint32_t* tile_counter, uint32_t* report_n, uint32_t* status,
                              int sm_count, cudaStream_t st);
// Crossing chains (longest first): their t values in cbuf.
void launch_chains(const GeomArgs& g, const int32_t* offs, const ChainWork& w, int32_t* cbuf, int sm_count,
                   cudaStream_t st);
// The records (curve, t bits) in the reference's order, from the chains.
void launch_order_records(const GeomArgs& g, const int32_t* offs, const ChainWork& w, const int32_t* cbuf, int2* rec,
                          uint32_t* status, int sm_count, cudaStream_t st);
// The same with the reference's flag bits (make_intersection_1.comp:361-375),
// for a read-back only.
void launch_merge(const GeomArgs& g, const int32_t* offs, const ChainWork& w, const int32_t* cbuf, int2* rec,
                  uint32_t* status, cudaStream_t st);
// One fragment per record: sort key + packed winding bits (4 bits: change,
// centre part).  With wnp NULL the bits are stored above the key bits of
// each key instead of in wnp[].
// n_cap launches the grid; the record count is read from n_dev (offs[C]).
struct SegArgs;
struct TileTables;
// seg: the per-path sort's segments (NULL: none), whose tables it builds when
// they are few (seg->tables_built).
void launch_fragment(const GeomArgs& g, const int2* rec, int64_t n_cap, const uint32_t* n_dev, uint64_t* keys,
                     uint8_t* wnp, DebugOut dbg, SegArgs* seg, uint32_t* status, cudaStream_t st);
TileTables segsort_tables(const SegArgs& a);

// ---- scan.cu
// Exclusive scan of n int32 values into out[0..n] (out[n] = total).  in and
// out may alias.  scratch: scan_scratch_bytes(n) bytes (0 for short inputs),
// no need to clear them.
size_t scan_scratch_bytes(int64_t n);
void launch_scan_i32(const int32_t* in, int32_t* out, int64_t n, void* scratch, cudaStream_t st);
// The same in a single pass with decoupled look-back (n > 0), as the frame's
// kernels scan: tile_status holds lookback_scan_words(n) zeroed words.
size_t lookback_scan_words(int64_t n);
void launch_lookback_scan_i32(const int32_t* in, int32_t* out, int64_t n, uint64_t* tile_status,
                              uint32_t* tile_counter, uint32_t* status, cudaStream_t st);

// ---- sort.cu  (onesweep LSD radix sort, 8-bit digits)
struct SortPlan {
    int64_t n;                 // element count, or the capacity when n_dev is set
    const uint32_t* n_dev;     // optional device-side count (<= n), read by the kernels
    uint32_t key_bits;
    uint32_t passes;
    uint32_t tiles;
    int items;                 // keys per thread of a tile: 8, 12 or 16
    int cleared = 0;           // 1: the caller has zeroed the scratch
    int hist_given = 0;        // 1: the digit counts are in the scratch (launch_row_starts), the rest zeroed
    // Where a wait of the sort gives up, it has left places of the order
    // unwritten, and the rows become empty: their starts (set by
    // launch_row_starts; NULL: none)
    int32_t* row_start = nullptr;
    uint32_t rows = 0;
};
SortPlan sort_plan(int64_t n, uint32_t key_bits, const uint32_t* n_dev = nullptr, int items = 12);
// Device scratch needed by a plan (bytes).
size_t sort_scratch_bytes(const SortPlan& p);
// Sorts (keys, values) stably by the low key_bits of the keys; higher bits
// travel with their key.  If vals_in is NULL the values are the identity
// 0..n-1; if vals_out is NULL there are no values (keys only).  Results end
// in (keys_out, vals_out); keys_alt/vals_alt are ping-pong buffers of n items.
void launch_sort_u64(const SortPlan& p, const uint64_t* keys_in, const uint32_t* vals_in, uint64_t* keys_out,
                     uint32_t* vals_out, uint64_t* keys_alt, uint32_t* vals_alt, void* scratch,
                     uint32_t* status, cudaStream_t st);
// The order of n draw records by row in one launch, where the rows and the
// records are few enough (after launch_row_starts; scratch: row_sort_bytes,
// zeroed).
bool row_sort_one_pass(int64_t n, uint32_t rows);
size_t row_sort_bytes(int64_t n, uint32_t rows);
void launch_row_sort(const uint32_t* rows_in, int64_t n, const uint32_t* n_dev, uint32_t rows, int32_t* row_start,
                     uint32_t* idx_out, void* scratch, uint32_t* status, cudaStream_t st);
// For a sort by row whose records per row are known: each row's first
// position row_start[0..rows] (exclusive scan; look-back words and counter
// zeroed) and every pass's digit counts into the plan's zeroed scratch, so
// that the sort needs no pass over the keys for them.
size_t row_scan_words(uint32_t rows);
void launch_row_starts(SortPlan& p, const uint32_t* row_count, uint32_t rows, int32_t* row_start, void* scratch,
                       uint64_t* tile_status, uint32_t* tile_counter, uint32_t* status, cudaStream_t st);
void launch_sort_u32(const SortPlan& p, const uint32_t* keys_in, const uint32_t* vals_in, uint32_t* keys_out,
                     uint32_t* vals_out, uint32_t* keys_alt, uint32_t* vals_alt, void* scratch,
                     uint32_t* status, cudaStream_t st);

// ---- segsort.cu  (stable sort of path-ordered keys: per-path segments)
// Segment p is the records of path p, from the paths' first curves and the
// curves' offsets.
struct SegArgs {
    const uint32_t* path_begin;   // [P + 1]
    const int32_t* offs;          // [C + 1]
    uint32_t n_paths;
    int64_t cap;                  // records the tables and buffers are sized for
    uint32_t max_size;            // > 0: a segment larger than that is flagged as a capacity overflow
    uint32_t* largest;            // largest segment of more than half a tile (0 if none); zeroed before
    uint32_t* wide_count;         // tiles that needed 64-bit items; zeroed before
    bool wide;                    // those tiles are sorted (else flagged as a capacity overflow)
    void* tables;                 // segsort_table_bytes
    void* zeroed;                 // segsort_zeroed_bytes, zeroed before
    bool tables_built = false;    // by launch_fragment
};
size_t segsort_table_bytes(uint32_t n_paths, int64_t cap);
size_t segsort_zeroed_bytes(uint32_t n_paths, int64_t cap);
int segsort_tile();
// Tiles of the sort with these tables, and of those the ones that needed
// 64-bit items (synchronous copies).
cudaError_t segsort_tile_counts(const SegArgs& a, uint32_t out[2]);
// The largest segment alone (before the sort's buffers exist).
void launch_segsort_largest(const SegArgs& a, cudaStream_t st);
// Sorts keys_in[0, N) into keys_out by their key bits (layout L; N from the
// offsets; cap bounds the tile tables); `levels` merge rounds launched, at
// least ceil(log2(chunks of the largest segment)).  keys_alt is scratch.
// The tile sort and the merge rounds run one wave of persistent CTAs.
// keys_in[0, N) is left unspecified (the tiles that need 64-bit items sort
// through it).
void launch_segsort(const SegArgs& a, uint64_t* keys_in, uint64_t* keys_out, uint64_t* keys_alt, const KeyLayout& L,
                    int levels, int sm_count, uint32_t* status, cudaStream_t st);

// ---- winding.cu
struct WindArgs {
    int64_t n;                      // N records: the capacity when n_dev is set
    const uint32_t* n_dev;          // device-side record count (offs[C])
    const uint64_t* skeys;          // sorted keys
    const uint32_t* svals;          // sorted record indices (NULL: winding bits ride in the keys)
    const uint8_t* wnp;             // packed winding bits by record index (NULL likewise)
    const uint32_t* fill_rule;      // [P]
    const uint32_t* fill_info;      // [P]
    uint32_t n_paths;
    int32_t W, H, F;
    int32_t pixel_mode;
    KeyLayout L;
    SceneTable st;
    int4* draw;                     // [capacity] paint runs {y << 16 | x, width, fill_info, 0}
    int64_t draw_capacity;
    uint32_t* draw_row;             // [capacity] global cell row of each paint run
    uint64_t* totals;               // [2] merged fragments, spans; zeroed before
    uint32_t* n_draw;               // [1] paint runs
    uint32_t* path_draw;            // [P] draw records per path (NULL unless labelling)
    // [cut_rows][cut_segs]: 1 + the last index of a run that covers a
    // resolve segment (kResolveSeg pixels) entirely and leaves nothing of
    // what was under it (an opaque one; pixel mode only);
    // zeroed before the emit
    uint32_t* seg_cut;
    uint32_t cut_rows, cut_segs;
    uint32_t* row_count;            // [cut_rows] paint runs per global cell row (zeroed before)
    unsigned long long* row_px;     // [cut_rows] pixels of a row's runs (widths summed; zeroed before)
    // parity dumps (NULL in production)
    int32_t* dbg_wscan;             // [N+1]
    int32_t* dbg_fflag;             // [N]
    int32_t* dbg_sflag;             // [N]
    int32_t* dbg_skey;              // [N]
};
// items: records per thread of a tile (4 or 8).  Look-back words (zeroed
// before), and words for the tiles' sums and prefixes; counters[0] (next
// tile) and counters[1] (tiles summed) are zeroed before.
size_t winding_status_words(int64_t n, int items = 8);
size_t winding_tile_words(int64_t n, int items = 8);
void launch_winding_emit(const WindArgs& a, int items, uint64_t* tile_status, uint64_t* tile_sums, uint32_t* counters,
                         uint32_t* status, cudaStream_t st);
// The reference's draw list (for a read-back), from the same sorted records
// and tile prefixes: draw records into a.draw; tile_status and counters[0]
// zeroed before.
void launch_draw_list(const WindArgs& a, int items, uint64_t* tile_status, const uint64_t* tile_sums,
                      uint32_t* counters, uint32_t* status, cudaStream_t st);

// ---- resolve.cu
// A gradient paint ready for the resolve (built on the host from an
// sr_paint and the scene's matrix, see sr.h for the definition): linear
// t = (lin0 X + lin1 Y) + lin2 of the pixel-space point (X, Y); radial
// g = (m0 X + m1 Y) + m2, (m3 X + m4 Y) + m5 in gradient space, focus
// (fx, fy), centre - focus (dx, dy), A = dx^2 + dy^2 - r^2.
constexpr int kMaxStops = 16;
struct DevPaint {
    int32_t kind, spread, n_stops, pad;
    float lin[3];
    float m[6];
    float fx, fy, dx, dy, A;
    float opacity;
    float off[kMaxStops];
    float rgba[kMaxStops][4];
};
// The paint a fill_info names: alpha byte 0 and index + 1 in the colour
// bytes; -1 for a solid colour.
__host__ __device__ __forceinline__ int32_t fill_paint(uint32_t info) {
    return (info >> 24) == 0u && (info & 0x00FFFFFFu) != 0u ? (int32_t)(info & 0x00FFFFFFu) - 1 : -1;
}

// Resolve work: a CTA paints segments or rows of one scene; cta_base[s] is the
// first CTA of scene s (host-built, n_scenes+1 entries).
struct ResolveArgs {
    const int4* draw;
    const uint32_t* row_sorted_idx;   // draw indices sorted by global cell row
    const int32_t* row_start;         // [total rows + 1]
    const uint32_t* cta_base;         // [n_scenes + 1]
    const SceneInfo* scenes;
    uint32_t n_scenes;
    int32_t F;
    int32_t pixel_mode;
    int32_t warps;                    // warps per CTA: 8 or 16
    int32_t seg;                      // pixels per warp: kResolveSeg, or 128 or 64
    uint32_t* image;                  // all scenes' RGBA8 framebuffers
    uint32_t* image2 = nullptr;       // the caller's memory for them too, or NULL
    const uint32_t* control = nullptr; // control block, whose first report_words words go to report (host memory)
    uint32_t* report = nullptr;
    uint32_t report_words = 0;
    const uint32_t* seg_cut;          // [rows][cut_segs] from the emit, or NULL
    const unsigned long long* row_px; // [rows] summed record widths from the emit, or NULL (every row searched)
    uint32_t cut_segs;
    const DevPaint* paints;           // gradient paints of the scene (single-scene contexts), or NULL
    uint32_t n_paints;
};
// Pixels per warp of the resolve (of a large frame), and of a cut.
constexpr int kResolveSeg = 256;
// Pixels per warp for a frame of `segs` segments of kResolveSeg pixels.
int resolve_segment(uint64_t segs, int pixel_mode, int sm_count);
// CTAs that a scene of `rows` cell rows takes.
uint32_t resolve_ctas(int32_t W, uint32_t rows, int seg, int warps);
void launch_resolve(const ResolveArgs& a, uint32_t n_ctas, cudaStream_t st);
// Multisampling: sum a sample frame into acc (first: start the sums), and
// write the rounded averages of k frames.
void launch_aa_accumulate(const uint32_t* img, void* acc, size_t n, bool first, cudaStream_t st);
// (img2: a second copy, or NULL)
void launch_aa_resolve(const void* acc, uint32_t* img, uint32_t* img2, size_t n, uint32_t k, cudaStream_t st);
// n pixels from a framebuffer to device memory of this device.
void launch_copy_image(const uint32_t* src, uint32_t* dst, size_t n, int sm_count, cudaStream_t st);
// n_dev (optional) holds the record count; n is the capacity.  With a status
// set by then (the sort gave up) every row is empty.
void launch_row_bounds(const uint32_t* srows, int64_t n, const uint32_t* n_dev, int32_t rows, int32_t* row_start,
                       const uint32_t* status, cudaStream_t st);

// ---- mlp.cu  (learned sizing: 6 features -> 64 -> 64 -> 2, GELU)
constexpr int kMlpIn = 6, kMlpHidden = 64, kMlpOut = 2;
constexpr int kMlpParams = kMlpHidden * kMlpIn + kMlpHidden + kMlpHidden * kMlpHidden + kMlpHidden +
                           kMlpOut * kMlpHidden + kMlpOut;
constexpr int kMlpNorm = 2 * kMlpIn + 2 * kMlpOut;
// feats[P][6] of the paths under the current transforms (tpos must be current).
void launch_path_features(const GeomArgs& g, const uint32_t* path_first_curve, uint32_t n_paths, float* feats,
                          cudaStream_t st);
// labels[P][2] = log(1 + records), log(1 + draw records) per path.
void launch_path_labels(const uint32_t* path_first_curve, uint32_t n_paths, const int32_t* count,
                        const uint32_t* path_draw, float* labels, cudaStream_t st);
// y[n][2] in log(1 + count) units.  wb: BF16 weights; master: FP32 copy (biases).
void launch_mlp_predict(const void* wb, const float* master, const float* norm, const float* x, uint32_t n, float* y,
                        int sm_count, cudaStream_t st);
// Adds the minibatch gradient of the mean squared error into grad and the
// sum of squared errors into loss_sum.
cudaError_t launch_mlp_grad(const void* wb, const float* master, const float* norm, const float* x, const float* t,
                            const uint32_t* idx, uint32_t n, float* grad, double* loss_sum, cudaStream_t st);
// A training step on n of the `rows` rows: the gradient, then Adam (by the last CTA of the same
// launch, which finds itself through `done`, a word zeroed before the first
// step); grad is zero before and after.
cudaError_t launch_mlp_step(void* wb, float* master, const float* norm, const float* x, const float* t,
                            const uint32_t* idx, uint32_t rows, uint32_t n, float* grad, double* loss_sum, float* m,
                            float* v, float lr, float b1, float b2, float eps, float bc1, float bc2, uint32_t* done,
                            cudaStream_t st);
void launch_to_bf16(const float* master, void* wb, cudaStream_t st);
void launch_perm_keys(uint32_t* keys, uint32_t n, uint64_t seed, cudaStream_t st);
// allot[P][2] from predictions with the path margins (margins[0..1]);
// frame capacities with the frame margins (margins[2..3]) accumulate into
// scene_tot[S][2] and tot[0..1], the allotments into tot[2..3] (zero them first).
void launch_allot(const float* y, uint32_t n_paths, const uint32_t* path_scene, const float margins[4],
                  uint32_t* allot, unsigned long long* scene_tot, unsigned long long* tot, cudaStream_t st);
// out[4] (zeroed first): paths over their record allotment, over their draw
// allotment, exact records, exact draw records.
void launch_judge(const uint32_t* path_first_curve, uint32_t n_paths, const int32_t* count, const uint32_t* path_draw,
                  const uint32_t* allot, unsigned long long* out, cudaStream_t st);

}  // namespace sr
