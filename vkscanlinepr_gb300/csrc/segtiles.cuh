// segtiles.cuh — the tables of the per-path sort (segsort.cu): which records
// each of its CTAs takes.  They need only the paths' record ranges, so in a
// frame of few paths the fragment kernel builds them with CTAs of its own.
#pragma once
#include "kernels.h"
#include "scan.cuh"

namespace sr {

constexpr int kTile = 4096;         // records a CTA sorts or merges
constexpr int kGroup = kTile / 2;   // largest segment packed into a group tile
constexpr uint32_t kChunkBit = 1u << 31;   // descriptor .z: a chunk of a large segment

// The tables of a frame: descriptors, in the table buffer, and what starts
// zeroed, in the zeroed buffer.
struct TileTables {
    uint4* desc;           // [max_tiles] {start, segment size, k | rounds << 16 | chunk bit, -}
    // [kMergeClasses][max_tiles] the chunk tiles of large segments by the merge
    // rounds their segment needs (1, 2, ...), in no order
    uint32_t* chunks;
    uint32_t mt;           // max_tiles
    uint32_t* fallback;    // [max_tiles] tiles left to the 64-bit tile sort, in no order
    uint32_t* tile_end;    // [max_tiles] end of a group tile (atomic max over its segments); zeroed
    uint64_t* scan_status; // look-back words of the tile scan; zeroed
    // zeroed: [0] scan counter, [2] next tile of the tile sort, [3] next of the
    // 64-bit sort, [4] tiles, [5 + l] next work item of merge round l, [16 + r]
    // chunk tiles of segments of r rounds
    uint32_t* ctl;
    uint32_t* wide_count;  // tiles left to the 64-bit sort
};
constexpr int kCtlSortNext = 2, kCtlFallbackNext = 3, kCtlTiles = 4, kCtlMergeNext = 5, kCtlChunks = 16;
constexpr uint32_t kMergeClasses = 5;   // the most rounds a frame takes
constexpr int kSegThreads = 128;   // segments a CTA of the tile scan takes

// Merge rounds a large segment of `chunks` sorted chunks needs.
SR_DEV uint32_t rounds_of(uint32_t chunks) {
    uint32_t r = 0;
    while ((1u << r) < chunks) ++r;
    return r;
}

// Records of path p: [a, e).
SR_DEV void seg_span(const SegArgs& s, uint32_t p, uint32_t& a, uint32_t& e) {
    a = (uint32_t)s.offs[s.path_begin[p]];
    e = (uint32_t)s.offs[s.path_begin[p + 1]];
}

// The largest segment of more than kGroup records.  max_size > 0: a segment
// larger than that is an overflow (the merge rounds of a pre-sized frame
// cannot take it; the frame is redone with exact sizing, which chooses the
// rounds, or the radix sort, from the largest segment).
SR_DEV void seg_note_size(const SegArgs& s, uint32_t size, uint32_t* status) {
    if (size > (uint32_t)kGroup) atomicMax(s.largest, size);
    if (s.max_size && size > s.max_size) set_error(status, ERR_CAPACITY);
}

// One pass over the segments (a thread each) for all tables: the tiles each
// segment opens (a large one its chunks, a small one that starts a group,
// i.e. the first small segment starting in its group, one tile), their
// exclusive scan, and the descriptors.  A group tile is opened by its head
// and stretched to the end of each small segment of the group.  Tiles past mt
// exist only in a frame whose records overflowed the capacity (it is redone);
// they are not written.
// (Segment starts, sizes, tiles, scan and descriptors used to be seven
// launches, 3.6-8 us each.)
SR_DEV void seg_tiles(const SegArgs& s, const TileTables& u, uint32_t* status, uint32_t spin_limit) {
    __shared__ uint32_t s_tile;
    __shared__ int32_t s_warp[kSegThreads / 32 + 1];
    const uint32_t mt = u.mt;
    if (threadIdx.x == 0) s_tile = atomicAdd(&u.ctl[0], 1u);
    __syncthreads();
    const uint32_t p = s_tile * kSegThreads + threadIdx.x;
    const bool live = p < s.n_paths;
    uint32_t a = 0, e = 0;
    int32_t n = 0;
    if (live) {
        seg_span(s, p, a, e);
        seg_note_size(s, e - a, status);
        if (e - a > (uint32_t)kGroup) {
            n = (int32_t)((e - a + kTile - 1) / kTile);
        } else {
            bool head = p == 0;
            if (!head) {
                const uint32_t pa = (uint32_t)s.offs[s.path_begin[p - 1]];
                head = a - pa > (uint32_t)kGroup || a / (uint32_t)kGroup != pa / (uint32_t)kGroup;
            }
            n = head ? 1 : 0;
        }
    }
    int32_t total;
    const int32_t first = scan_thread_values<kSegThreads>(n, s_tile, u.scan_status, status, spin_limit, s_warp, &total);
    if (!live) return;
    if (p == s.n_paths - 1) u.ctl[kCtlTiles] = (uint32_t)total;
    if (e - a > (uint32_t)kGroup) {
        const uint32_t rounds = rounds_of((uint32_t)n);
        const int32_t m = (int32_t)min((uint32_t)n, mt - min(mt, (uint32_t)first));   // chunks that fit the table
        // (more rounds than that only in a frame that is redone)
        const uint32_t cls = min(rounds, kMergeClasses);
        const uint32_t at = cls && m > 0 ? atomicAdd(&u.ctl[kCtlChunks + cls], (uint32_t)m) : 0u;
        for (int32_t k = 0; k < m; ++k) {
            u.desc[first + k] = make_uint4(a, e - a, (uint32_t)k | (rounds << 16) | kChunkBit, 0u);
            // (more than mt of a class only where a wait gave up and `first` is wrong)
            if (cls && at + (uint32_t)k < mt) u.chunks[(size_t)(cls - 1) * mt + at + k] = (uint32_t)(first + k);
        }
        return;
    }
    // a non-head small segment belongs to the tile opened just before it
    const int32_t tile = n == 1 ? first : first - 1;
    if (tile < 0 || (uint32_t)tile >= mt) return;
    if (n == 1) u.desc[tile] = make_uint4(a, 0u, 0u, 0u);
    // (without records it ends where it starts: 2 million such paths, all at one
    // word, took 1.3 ms)
    if (e > a) atomicMax(&u.tile_end[tile], e);
}

}  // namespace sr
