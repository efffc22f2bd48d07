// resolve.cu — paints the draw list into the RGBA8 framebuffer.
//
// Replaces the reference's graphics pass (scanlinepr.vert:18-51,
// scanlinepr.frag:7-14, pipeline at scanline_rasterizer.cpp:881-944 and
// :610-695): each draw record (yx, width, colour, index) covers
// [x, x+width) x [y, y+FRAG_SIZE), the framebuffer is cleared to white, and
// records land in draw order.  Reference mode overwrites (blending is off in
// the reference pipeline); pixel mode composites source-over with integer
// arithmetic.  Draw records are first sorted stably by cell row (onesweep), so
// a row's records are applied in path order; a thread owns a fixed set of
// pixels, so no barrier is needed between records.  A warp paints a segment of a
// row: in pixel mode it first finds where its painting may start (the collapse
// cut below), in reference mode it takes the latest record of each pixel.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace sr {

// First index of every cell row in the row-sorted draw list.
__global__ void k_row_bounds(const uint32_t* __restrict__ srows, int64_t n_cap, const uint32_t* __restrict__ n_dev,
                             int32_t rows, int32_t* __restrict__ row_start, const uint32_t* __restrict__ status) {
    if (*status) {   // the order has places that nobody wrote
        const int32_t step = (int32_t)(gridDim.x * blockDim.x);
        for (int32_t r = (int32_t)(blockIdx.x * blockDim.x + threadIdx.x); r <= rows; r += step) row_start[r] = 0;
        return;
    }
    const int64_t n = n_dev ? (int64_t)min((uint64_t)*n_dev, (uint64_t)n_cap) : n_cap;
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i <= n; i += stride) {
        int32_t cur = i < n ? (int32_t)srows[i] : rows;
        uint32_t pv = i > 0 ? srows[i - 1] : 0xFFFFFFFFu;
        int32_t prev = pv == 0xFFFFFFFFu ? -1 : (int32_t)(pv > (uint32_t)rows ? (uint32_t)rows : pv);
        if ((uint32_t)cur > (uint32_t)rows) cur = rows;
        for (int32_t r = prev + 1; r <= cur; ++r) row_start[r] = (int32_t)i;
    }
}

// ----------------------------------------------------------- pixel mode --
// Source-over in path order over opaque white: for R, G, B
//   c' = floor((s*a + c*(255-a) + 127) / 255) = round((s*a + c*(255-a)) / 255).
// Red and blue share one 32-bit word (r in bits 0-7, b in bits 16-23) and
// blend with integer operations: u = c*ia + s*a + 128 fits each 16-bit
// half (<= 65153), and c' = (u + (u >> 8)) >> 8 per half, the two shifts
// being byte permutes (bytes 1 and 3 to 0 and 2); no half carries into the
// other.  Green blends on the FMA pipe: u = c*ia + s*a is an exact float
// (<= 65025), and fma(u, 1/255, 1.5*2^23) - 1.5*2^23 rounds u/255 to the
// nearest integer.  Both forms equal the formula for every reachable u
// (checked exhaustively by the CPU tests).  Alpha stays 255:
// (255*a + 255*(255-a) + 127) / 255 = 255.
constexpr float kRound = 12582912.0f;   // 1.5 * 2^23
constexpr int kChunk = 1024;
constexpr uint64_t kHalfSegs = 200, kQuarterSegs = 40;   // segments of kResolveSeg an SM

struct PixRec {
    int32_t x0, x1;     // [x0, x1) clipped to >= 0
    float ia;           // 255 - a
    float sg;           // s*a of green
    uint32_t iau;       // 255 - a
    uint32_t sab;       // (s*a + 128) of red | of blue << 16
    uint32_t pad;       // 32 bytes: two 16-byte accesses
    uint32_t idx1;      // 1 + draw index
};

// q: a record's iau, sab, ia and sg (a PixRec or a RunRec).
template <class Rec> SR_DEV void blend3(uint32_t& rb, float& g, const Rec& q) {
    const uint32_t u = rb * q.iau + q.sab;
    rb = __byte_perm(u + __byte_perm(u, 0u, 0x4341u), 0u, 0x4341u);
    const float ug = __fmaf_rn(g, q.ia, q.sg);
    g = __fsub_rn(__fmaf_rn(ug, 1.0f / 255.0f, kRound), kRound);
}

int resolve_segment(uint64_t segs, int pixel_mode, int sm_count) {
    const uint64_t sms = (uint64_t)(sm_count > 0 ? sm_count : 1);
    if (segs >= (pixel_mode ? kHalfSegs : kQuarterSegs) * sms) return kResolveSeg;
    return segs >= kQuarterSegs * sms ? kResolveSeg / 2 : kResolveSeg / 4;
}

uint32_t resolve_ctas(int32_t W, uint32_t rows, int seg, int warps) {
    const uint32_t segs = (uint32_t)((W + seg - 1) / seg);
    return (rows * segs + (uint32_t)warps - 1) / (uint32_t)warps;
}

SR_DEV uint32_t scene_of_cta(const ResolveArgs& a) {   // last s with cta_base[s] <= blockIdx.x
    uint32_t lo = 0, hi = a.n_scenes;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (a.cta_base[mid] <= blockIdx.x) lo = mid;
        else hi = mid;
    }
    return lo;
}

// A warp skips the records before the last one that covers its whole segment
// and hides what is under it (seg_cut, written by the emit): source-over with
// a = 255 gives floor((255 s + 127) / 255) = s whatever the pixel held.
SR_DEV uint32_t resolve_cut(const ResolveArgs& a, uint32_t global_row, int32_t seg) {
    return a.seg_cut ? a.seg_cut[(size_t)global_row * a.cut_segs + (uint32_t)(seg / kResolveSeg)] : 0u;
}

// Colour of gradient paint P at the pixel-space point (x, y), packed RGBA8,
// 0 when transparent (the definition is in sr.h; the oracle restates it).
__device__ __noinline__ uint32_t paint_color(const DevPaint& P, float x, float y) {
    float t;
    if (P.kind == 1) {
        t = __fadd_rn(__fadd_rn(__fmul_rn(P.lin[0], x), __fmul_rn(P.lin[1], y)), P.lin[2]);
    } else {
        const float gx = __fadd_rn(__fadd_rn(__fmul_rn(P.m[0], x), __fmul_rn(P.m[1], y)), P.m[2]);
        const float gy = __fadd_rn(__fadd_rn(__fmul_rn(P.m[3], x), __fmul_rn(P.m[4], y)), P.m[5]);
        const float ex = __fsub_rn(gx, P.fx), ey = __fsub_rn(gy, P.fy);
        const float b = __fadd_rn(__fmul_rn(ex, P.dx), __fmul_rn(ey, P.dy));
        const float c = __fadd_rn(__fmul_rn(ex, ex), __fmul_rn(ey, ey));
        if (P.A == 0.0f) {
            t = b != 0.0f ? __fdiv_rn(c, __fmul_rn(2.0f, b)) : 0.0f;
        } else {
            const float disc = __fsub_rn(__fmul_rn(b, b), __fmul_rn(P.A, c));
            if (disc < 0.0f) {
                t = 0.0f;
            } else {
                const float sq = __fsqrt_rn(disc);
                t = __fdiv_rn(P.A < 0.0f ? __fsub_rn(b, sq) : __fadd_rn(b, sq), P.A);
            }
        }
    }
    if (!(t == t)) t = 0.0f;
    if (P.spread == 1) {
        t = __fsub_rn(t, floorf(t));
    } else if (P.spread == 2) {
        const float u = __fsub_rn(t, __fmul_rn(2.0f, floorf(__fmul_rn(t, 0.5f))));
        t = u > 1.0f ? __fsub_rn(2.0f, u) : u;
    } else {
        t = gmin(gmax(t, 0.0f), 1.0f);
    }
    const int n = P.n_stops;
    if (n <= 0) return 0u;
    float ch[4];
    if (!(t > P.off[0])) {
#pragma unroll
        for (int q = 0; q < 4; ++q) ch[q] = P.rgba[0][q];
    } else if (!(t < P.off[n - 1])) {
#pragma unroll
        for (int q = 0; q < 4; ++q) ch[q] = P.rgba[n - 1][q];
    } else {
        int k = 0;
        while (k + 2 < n && !(t < P.off[k + 1])) ++k;
        const float f = __fdiv_rn(__fsub_rn(t, P.off[k]), __fsub_rn(P.off[k + 1], P.off[k]));
#pragma unroll
        for (int q = 0; q < 4; ++q) ch[q] = lerp_rn(P.rgba[k][q], P.rgba[k + 1][q], f);
    }
    ch[3] = __fmul_rn(ch[3], P.opacity);
    uint32_t col = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        float v = __fmul_rn(ch[q], 255.0f);
        if (!(v > 0.0f)) v = 0.0f;
        if (v > 255.0f) v = 255.0f;
        col |= (uint32_t)v << (8 * q);
    }
    return (col >> 24) ? col : 0u;
}

// A gradient record's PixRec carries iau = kGradient and its paint in sab.
constexpr uint32_t kGradient = 0xFFFFFFFFu;

SR_DEV PixRec solid_rec(uint32_t col) {
    PixRec pr;
    const uint32_t al = col >> 24;
    pr.ia = (float)(255u - al);
    pr.sg = (float)(((col >> 8) & 0xFFu) * al);
    pr.iau = 255u - al;
    pr.sab = ((col & 0xFFu) * al + 128u) | ((((col >> 16) & 0xFFu) * al + 128u) << 16);
    return pr;
}

// GRAD: the kernel paints gradients.  Without it a gradient record is a
// solid of alpha 0, which leaves every pixel as it was; the kernels without
// gradients run for scenes without paints and keep their registers.
template <bool GRAD> SR_DEV PixRec pix_rec(const int4 d, uint32_t di) {
    PixRec pr;
    pr.idx1 = di + 1u;
    const int32_t x = d.x & 0xFFFF;
    pr.x0 = x;
    pr.x1 = wadd(x, d.y);
    const uint32_t col = (uint32_t)d.z, al = col >> 24;
    const int32_t paint = GRAD ? fill_paint(col) : -1;
    if (paint >= 0) {
        pr.iau = kGradient;
        pr.sab = (uint32_t)paint;
        pr.ia = 0.0f;
        pr.sg = 0.0f;
        pr.pad = 0;
        return pr;
    }
    pr.ia = (float)(255u - al);
    pr.sg = (float)(((col >> 8) & 0xFFu) * al);
    pr.iau = 255u - al;
    pr.sab = ((col & 0xFFu) * al + 128u) | ((((col >> 16) & 0xFFu) * al + 128u) << 16);
    pr.pad = 0;
    return pr;
}

// A gradient record: each lane blends its covered pixels with the paint's
// colour at their centres (row centre yc); a paint the table lacks paints
// nothing.
template <int K>
SR_DEV void apply_gradient(const ResolveArgs& a, const PixRec& pr, int32_t seg, int lane, float yc,
                           uint32_t (&rb)[K], float (&g)[K]) {
    if (!a.paints || pr.sab >= a.n_paints) return;
    const DevPaint& P = a.paints[pr.sab];
#pragma unroll
    for (int j = 0; j < K; ++j) {
        const int32_t p = seg + lane + 32 * j;
        if (p >= pr.x0 && p < pr.x1) {
            const uint32_t col = paint_color(P, __fadd_rn((float)p, 0.5f), yc);
            if (col) blend3(rb[j], g[j], solid_rec(col));
        }
    }
}

// A record on this warp's segment: a one-pixel record is a uniform branch on
// its register slot; a record over the whole segment blends every slot;
// otherwise each lane tests its pixels.
template <bool GRAD, int K>
SR_DEV void apply_pix(const ResolveArgs& a, const PixRec& pr, int32_t seg, int lane, float yc, uint32_t (&rb)[K],
                      float (&g)[K]) {
    if (GRAD && pr.iau == kGradient) {
        apply_gradient(a, pr, seg, lane, yc, rb, g);
    } else if (K == 8 && pr.x1 - pr.x0 == 1) {
        const int32_t off = pr.x0 - seg;
        const int j = off >> 5;
        if (lane == (off & 31)) {
            switch (j) {
                case 0: blend3(rb[0], g[0], pr); break;
                case 1: blend3(rb[1 % K], g[1 % K], pr); break;
                case 2: blend3(rb[2 % K], g[2 % K], pr); break;
                case 3: blend3(rb[3 % K], g[3 % K], pr); break;
                case 4: blend3(rb[4 % K], g[4 % K], pr); break;
                case 5: blend3(rb[5 % K], g[5 % K], pr); break;
                case 6: blend3(rb[6 % K], g[6 % K], pr); break;
                default: blend3(rb[7 % K], g[7 % K], pr); break;
            }
        }
    } else if (pr.x0 <= seg && pr.x1 >= seg + 32 * K) {
#pragma unroll
        for (int j = 0; j < K; ++j) blend3(rb[j], g[j], pr);
    } else {
#pragma unroll
        for (int j = 0; j < K; ++j) {
            int32_t p = seg + lane + 32 * j;
            if (p >= pr.x0 && p < pr.x1) blend3(rb[j], g[j], pr);
        }
    }
}

// Where a segment's painting may start.  Every pixel-blend is monotone in
// the pixel's old value (c' = floor((s*a + c*(255-a) + 127) / 255)), and so
// is any composition of them.  If a run of records that each cover the whole
// segment maps 0 and 255 to the same value in R, G and B, it maps every
// value there: the segment holds one colour after the run whatever it held
// before, so painting from white at the run's first record gives the same
// pixels as painting from the row's first record.  With alpha >= 0.4 a run
// of a handful of layers usually does this; an opaque span is a run of one.
// A warp walks the last kChunk records of its row from the end back,
// collects each run of whole-segment records between records that cover
// only part of the segment (the latest 32 of a longer run), and lane t
// tests the run's suffix from its record t: the latest start that collapses
// is the cut.  Without one the segment is painted from the row's start.
// The walk costs about a pass over the records it reads, so it is skipped
// for rows of fewer than kSearchLayers layers a pixel (record widths summed
// by the emit, over the row's width): a cut needs a run of several whole-
// segment layers and saves little there.
constexpr unsigned kSearchLayers = 32;

SR_DEV bool row_searched(const ResolveArgs& a, uint32_t r, int32_t W) {
    return !a.row_px || a.row_px[r] >= (unsigned long long)kSearchLayers * (unsigned long long)W;
}

struct RunRec {
    uint32_t iau, sab;
    float ia, sg;
};

SR_DEV RunRec run_rec(const PixRec& p) {
    RunRec r;
    r.iau = p.iau;
    r.sab = p.sab;
    r.ia = p.ia;
    r.sg = p.sg;
    return r;
}

// A warp's run of whole-segment records, in draw order with the latest at
// [31], and their positions.
struct RunBuf {
    RunRec rec[32];
    int32_t pos[32];
};

// The latest position among the n held records from which the run to [31]
// sends 0 and 255 to one colour, or -1.
SR_DEV int32_t run_collapse(const RunBuf& buf, int n, int lane) {
    uint32_t lo_rb = 0u, hi_rb = 0x00FF00FFu;
    float lo_g = 0.0f, hi_g = 255.0f;
    for (int k = 32 - n; k < 32; ++k) {
        const RunRec r = buf.rec[k];
        if (k >= lane) {
            blend3(lo_rb, lo_g, r);
            blend3(hi_rb, hi_g, r);
        }
    }
    const uint32_t m = __ballot_sync(0xFFFFFFFFu, lane >= 32 - n && lo_rb == hi_rb && lo_g == hi_g);
    return m ? buf.pos[31 - __clz(m)] : -1;
}

// The run bookkeeping of a backward walk: feed() takes 32 records at a time
// (latest lane first), each overlapping the segment or not and covering all
// of it or not.
struct RunWalk {
    int n = 0;          // records of the current run held
    bool full = false;  // the held run filled the buffer and did not collapse
    int32_t cut = -1;

    // Returns true once a cut is found.  Covers above the highest record
    // over part of the segment extend the current run; that record ends it;
    // the covers below it start the next run, and so on.  A run's records
    // enter the buffer together, each lane at its rank from the top.
    SR_DEV bool feed(uint32_t mo, uint32_t mc, const PixRec& mine, int32_t pos, int lane, RunBuf& buf) {
        uint32_t mp = mo & ~mc;
        for (;;) {
            const uint32_t above = mp ? ~((2u << (31 - __clz(mp))) - 1u) : 0xFFFFFFFFu;
            const uint32_t run = mc & above;
            if (run && !full) {
                const int rank = n + __popc(run & ~((2u << lane) - 1u));
                if (((run >> lane) & 1u) && rank < 32) {
                    buf.rec[31 - rank] = run_rec(mine);
                    buf.pos[31 - rank] = pos;
                }
                __syncwarp();
                n += __popc(run);
                if (n >= 32) {
                    n = 32;
                    cut = run_collapse(buf, n, lane);
                    if (cut >= 0) return true;
                    full = true;
                }
            }
            if (!mp) return false;
            if (close(lane, buf)) return true;
            mc &= ~above;
            mp &= ~above & ((1u << (31 - __clz(mp))) - 1u);
            if (!mc) return false;
        }
    }

    SR_DEV bool close(int lane, RunBuf& buf) {
        if (n && !full) {
            cut = run_collapse(buf, n, lane);
            if (cut >= 0) return true;
        }
        n = 0;
        full = false;
        return false;
    }
};

template <int K> SR_DEV void init_pix(uint32_t (&rb)[K], float (&g)[K]) {
#pragma unroll
    for (int j = 0; j < K; ++j) {
        rb[j] = 0x00FF00FFu;
        g[j] = 255.0f;
    }
}

// The row's pixels into the framebuffer, and into the caller's (a copy of the
// framebuffer would read it again, and be one more launch).
template <int K>
SR_DEV void store_pix(const ResolveArgs& a, uint64_t row, int32_t W, int32_t seg, int lane, const uint32_t (&rb)[K],
                      const float (&g)[K]) {
#pragma unroll
    for (int j = 0; j < K; ++j) {
        int32_t p = seg + lane + 32 * j;
        if (p < W) {
            const uint32_t v = rb[j] | ((uint32_t)__float2int_rn(g[j]) << 8) | 0xFF000000u;
            a.image[row + (uint32_t)p] = v;
            if (a.image2) a.image2[row + (uint32_t)p] = v;
        }
    }
}

// The frame's report: the control block's first words into page-locked host
// memory (every kernel that writes them is done), for the wait at the frame's
// end; a copy of its own would be one more launch.
SR_DEV void write_report(const ResolveArgs& a) {
    if (blockIdx.x == 0 && threadIdx.x < a.report_words) a.report[threadIdx.x] = a.control[threadIdx.x];
}

// A warp paints one segment of one row, by itself: it finds its cut and
// streams the row's records from there, 32 at a time, through its own
// shared-memory slots.  The warps of a CTA mostly share a row, so the records
// come from L1, and no warp waits for another.  (A CTA a row that staged the
// row's last 1,024 records for its warps, beside a kernel like this one for
// canvases narrower than the CTA, each with a grid over all rows: 0.160 ms for
// the 4096^2 frame and 0.70 for 64 uneven scenes, against 0.121 and 0.50.
// Blank canvases took 0.257 of the 0.70, now 0.131.)  Instructions bound it,
// some 20 a record and 7 a record and 32 pixels, and in a small frame the
// latency of a row's records one after the other.
//
// So a warp's segment is shorter when the frame has few: 256 pixels, 128 below
// 200 such segments an SM, 64 below 40.  With 256 / 128 / 64 the kernel took,
// in ms: 4096^2 frame of 20,000 paths (431 segments an SM) 0.121 / 0.188 /
// 0.354, 2048^2 frame of 5,000 (108) 0.078 / 0.060 / 0.076, of 3,000 stars
// 0.070 / 0.060 / 0.078, 1024^2 frame of 3,000 (27) 0.109 / 0.080 / 0.059, of
// 500 stars 0.0184 / 0.0164 / 0.0164, 512^2 frame of 3,000 0.144 / 0.106 /
// 0.076, 256^2 frame of 3,000 0.301 / 0.180 / 0.147.  (Chosen by the scene in a
// batch, the narrow ones at 128: 0.51 instead of 0.50.)
template <int WARPS, int K, bool GRAD>
__global__ void __launch_bounds__(32 * WARPS, (GRAD ? 32 : K == 8 ? 40 : 48) / WARPS) k_resolve_pixel(const ResolveArgs a) {
    wait_for_stream();
    write_report(a);
    constexpr int kSeg = 32 * K;
    static_assert(kResolveSeg % kSeg == 0, "a cut covers whole segments");
    __shared__ PixRec slots[WARPS * 32];
    __shared__ RunBuf bufs[WARPS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t scene = scene_of_cta(a);
    const SceneInfo* si = &a.scenes[scene];
    const int32_t W = si->W;
    const uint32_t segs = (uint32_t)(W + kSeg - 1) / kSeg;
    const uint32_t item = (blockIdx.x - a.cta_base[scene]) * WARPS + (uint32_t)warp;
    const uint32_t y = item / segs;
    if (y >= si->rows) return;
    const int32_t seg = (int32_t)(item - y * segs) * kSeg;
    PixRec* slot = slots + warp * 32;
    RunBuf& buf = bufs[warp];
    const uint32_t r = si->row_base + y;
    const int32_t beg = a.row_start[r], end = a.row_start[r + 1];
    const int32_t segend = imin(seg + kSeg, W);
    const uint32_t cut = resolve_cut(a, r, seg);
    int32_t start = beg;
    if (row_searched(a, r, W)) {
        RunWalk rw;
        const int32_t lim = imax(beg, end - kChunk);
        bool found = false;
        for (int32_t c1 = end; c1 > lim && !found; c1 -= 32) {
            const int32_t q = c1 - 32 + lane;
            bool ov = false, cover = false;
            PixRec pr;
            if (q >= lim) {
                const uint32_t di = a.row_sorted_idx[q];
                pr = pix_rec<GRAD>(a.draw[di], di);
                ov = pr.x0 < seg + kSeg && pr.x1 > seg;
                // a gradient's colour varies over the segment: it ends a run
                cover = pr.x0 <= seg && pr.x1 >= segend && pr.iau != kGradient;
            }
            found = rw.feed(__ballot_sync(0xFFFFFFFFu, ov), __ballot_sync(0xFFFFFFFFu, cover), pr, q, lane, buf);
        }
        if (found || rw.close(lane, buf)) start = rw.cut;
    }
    uint32_t rb[K];
    float g[K];
    init_pix<K>(rb, g);
    const float yc = __fadd_rn((float)y, 0.5f);
    for (int32_t c0 = start; c0 < end; c0 += 32) {
        const int32_t q = c0 + lane;
        bool ov = false;
        if (q < end) {
            const uint32_t di = a.row_sorted_idx[q];
            const PixRec pr = pix_rec<GRAD>(a.draw[di], di);
            ov = pr.x0 < seg + kSeg && pr.x1 > seg && pr.idx1 >= cut;
            if (ov) slot[lane] = pr;
        }
        uint32_t m = __ballot_sync(0xFFFFFFFFu, ov);
        __syncwarp();
        while (m) {
            const PixRec p = slot[__ffs(m) - 1];
            m &= m - 1;
            apply_pix<GRAD, K>(a, p, seg, lane, yc, rb, g);
        }
        __syncwarp();
    }
    store_pix<K>(a, si->image_off + (uint64_t)y * (uint32_t)W, W, seg, lane, rb, g);
}

// ------------------------------------------------------- reference mode --
// Overwrite in draw order (blending off); a cell row is FRAG_SIZE pixel rows,
// painted alike.  A pixel takes the latest record over it, so a warp walks its
// row's records from the end back, 32 at a time, fills the pixels of its segment
// that have none yet and stops when all have.  (A CTA a row or several short
// ones that staged all their records for its warps, in draw order, took 18 us for
// a 1000x750 frame of 1,200 paths and 82 for the 4096^2 one; this takes 8 and 43.)
// 64 pixels a warp below 40 segments of 256 an SM, else 256: for 512^2 and 3,000
// paths 8 us with 64 and 12 with 256, for 2048^2 and 5,000 24 and 18 (128: 20).
struct RefRec {
    int32_t x0, x1;
    uint32_t col;
};

template <int WARPS, int K, bool GRAD>
__global__ void __launch_bounds__(32 * WARPS) k_resolve_ref(const ResolveArgs a) {
    wait_for_stream();
    write_report(a);
    constexpr int kSeg = 32 * K;
    __shared__ RefRec slots[WARPS * 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t scene = scene_of_cta(a);
    const SceneInfo* si = &a.scenes[scene];
    const int32_t W = si->W;
    const uint32_t segs = (uint32_t)(W + kSeg - 1) / kSeg;
    const uint32_t item = (blockIdx.x - a.cta_base[scene]) * WARPS + (uint32_t)warp;
    const uint32_t y = item / segs;
    if (y >= si->rows) return;
    const int32_t seg = (int32_t)(item - y * segs) * kSeg;
    RefRec* slot = slots + warp * 32;
    const uint32_t r = si->row_base + y;
    const int32_t beg = a.row_start[r], end = a.row_start[r + 1];
    uint32_t px[K], open = 0;   // pixels on the canvas without a record yet
#pragma unroll
    for (int j = 0; j < K; ++j) {
        px[j] = 0xFFFFFFFFu;
        open |= (seg + lane + 32 * j < W ? 1u : 0u) << j;
    }
    for (int32_t c1 = end; c1 > beg && __any_sync(0xFFFFFFFFu, open != 0); c1 -= 32) {
        const int32_t q = c1 - 32 + lane;
        bool ov = false;
        if (q >= beg) {
            const int4 d = a.draw[a.row_sorted_idx[q]];
            const int32_t x0 = d.x & 0xFFFF, x1 = wadd(x0, d.y);
            ov = x0 < seg + kSeg && x1 > seg && div_F(d.x >> 16, a.F) == (int32_t)y;
            // a gradient that the table lacks paints nothing
            if (GRAD && ov && fill_paint((uint32_t)d.z) >= 0)
                ov = a.paints && (uint32_t)fill_paint((uint32_t)d.z) < a.n_paints;
            if (ov) slot[lane] = RefRec{x0, x1, (uint32_t)d.z};
        }
        uint32_t m = __ballot_sync(0xFFFFFFFFu, ov);
        __syncwarp();
        while (m) {
            const int b = 31 - __clz((int)m);
            m &= ~(1u << b);
            const RefRec rr = slot[b];
            const int32_t paint = GRAD ? fill_paint(rr.col) : -1;
            // a gradient is sampled on the cell's centre row
            const float yc = GRAD ? __fadd_rn((float)((int32_t)y * a.F), 1.0f) : 0.0f;
#pragma unroll
            for (int j = 0; j < K; ++j) {
                const int32_t p = seg + lane + 32 * j;
                if (((open >> j) & 1u) && p >= rr.x0 && p < rr.x1) {
                    px[j] = paint >= 0 ? paint_color(a.paints[paint], __fadd_rn((float)p, 0.5f), yc) : rr.col;
                    open &= ~(1u << j);
                }
            }
        }
        __syncwarp();
    }
    const int32_t y0 = (int32_t)y * a.F, nrows = imin(a.F, si->H - y0);
    for (int32_t yy = 0; yy < nrows; ++yy) {
        const uint64_t row = si->image_off + (uint64_t)(y0 + yy) * (uint32_t)W;
#pragma unroll
        for (int j = 0; j < K; ++j) {
            const int32_t p = seg + lane + 32 * j;
            if (p < W) {
                a.image[row + (uint32_t)p] = px[j];
                if (a.image2) a.image2[row + (uint32_t)p] = px[j];
            }
        }
    }
}

template <int WARPS, bool GRAD> static void launch_resolve_t(const ResolveArgs& a, uint32_t n_ctas, cudaStream_t st) {
    if (a.pixel_mode) {
        if (a.seg == 64) launch_after(k_resolve_pixel<WARPS, 2, GRAD>, n_ctas, 32 * WARPS, 0, st, a);
        else if (a.seg == 128) launch_after(k_resolve_pixel<WARPS, 4, GRAD>, n_ctas, 32 * WARPS, 0, st, a);
        else launch_after(k_resolve_pixel<WARPS, 8, GRAD>, n_ctas, 32 * WARPS, 0, st, a);
    } else {
        if (a.seg == kResolveSeg / 4) launch_after(k_resolve_ref<WARPS, 2, GRAD>, n_ctas, 32 * WARPS, 0, st, a);
        else launch_after(k_resolve_ref<WARPS, 8, GRAD>, n_ctas, 32 * WARPS, 0, st, a);
    }
}

void launch_resolve(const ResolveArgs& a, uint32_t n_ctas, cudaStream_t st) {
    if (n_ctas == 0) return;
    count_launches(1);
    const bool grad = a.paints && a.n_paints;
    if (a.warps == 8) {
        if (grad) launch_resolve_t<8, true>(a, n_ctas, st);
        else launch_resolve_t<8, false>(a, n_ctas, st);
    } else {
        if (grad) launch_resolve_t<16, true>(a, n_ctas, st);
        else launch_resolve_t<16, false>(a, n_ctas, st);
    }
}

// Multisampling: the sample frames summed per channel (ushort4; 16 samples
// of 255 fit), then the rounded average (sum + k/2) / k per channel.
__global__ void k_aa_accumulate(const uint32_t* __restrict__ img, ushort4* __restrict__ acc, size_t n, int first) {
    wait_for_stream();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t c = img[i];
    ushort4 v = first ? make_ushort4(0, 0, 0, 0) : acc[i];
    v.x = (unsigned short)(v.x + (c & 0xFFu));
    v.y = (unsigned short)(v.y + ((c >> 8) & 0xFFu));
    v.z = (unsigned short)(v.z + ((c >> 16) & 0xFFu));
    v.w = (unsigned short)(v.w + (c >> 24));
    acc[i] = v;
}

__global__ void k_aa_resolve(const ushort4* __restrict__ acc, uint32_t* __restrict__ img, uint32_t* __restrict__ img2,
                             size_t n, uint32_t k) {
    wait_for_stream();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const ushort4 v = acc[i];
    const uint32_t h = k / 2u;
    const uint32_t c = ((v.x + h) / k) | (((v.y + h) / k) << 8) | (((v.z + h) / k) << 16) | (((v.w + h) / k) << 24);
    img[i] = c;
    if (img2) img2[i] = c;
}

// A framebuffer to the caller's device memory: four 16-byte loads in flight a
// thread, or 4-byte ones where either lies off 16 bytes.  The 64 images (423
// MB) of a batch take 228 us, a launch each (3.5 us of host time), where
// cudaMemcpyAsync took 687.
template <class T>
__global__ void __launch_bounds__(256) k_copy(const T* __restrict__ src, T* __restrict__ dst, size_t n) {
    wait_for_stream();
    const size_t stride = (size_t)gridDim.x * 1024;
    for (size_t i = (size_t)blockIdx.x * 1024 + threadIdx.x; i < n; i += stride) {
        T v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (i + 256 * k < n) v[k] = src[i + 256 * k];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (i + 256 * k < n) dst[i + 256 * k] = v[k];
    }
}

void launch_aa_accumulate(const uint32_t* img, void* acc, size_t n, bool first, cudaStream_t st) {
    if (!n) return;
    count_launches(1);
    launch_after(k_aa_accumulate, (unsigned)((n + 255) / 256), 256, 0, st, img, static_cast<ushort4*>(acc), n,
                 first ? 1 : 0);
}

void launch_aa_resolve(const void* acc, uint32_t* img, uint32_t* img2, size_t n, uint32_t k, cudaStream_t st) {
    if (!n) return;
    count_launches(1);
    launch_after(k_aa_resolve, (unsigned)((n + 255) / 256), 256, 0, st, static_cast<const ushort4*>(acc), img, img2, n,
                 k);
}

void launch_copy_image(const uint32_t* src, uint32_t* dst, size_t n, int sm_count, cudaStream_t st) {
    if (!n) return;
    count_launches(1);
    const bool vec = ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15u) == 0 && n % 4 == 0;
    const size_t items = vec ? n / 4 : n;
    const unsigned grid = (unsigned)std::min<size_t>((items + 1023) / 1024, (size_t)std::max(sm_count, 1) * 8);
    if (vec)
        launch_after(k_copy<uint4>, grid, 256, 0, st, reinterpret_cast<const uint4*>(src),
                     reinterpret_cast<uint4*>(dst), items);
    else
        launch_after(k_copy<uint32_t>, grid, 256, 0, st, src, dst, items);
}

void launch_row_bounds(const uint32_t* srows, int64_t n, const uint32_t* n_dev, int32_t rows, int32_t* row_start,
                       const uint32_t* status, cudaStream_t st) {
    int64_t work = n + 1;
    int blocks = (int)((work + 255) / 256);
    if (blocks > 1216) blocks = 1216;
    count_launches(1);
    k_row_bounds<<<blocks, 256, 0, st>>>(srows, n, n_dev, rows, row_start, status);
}

}  // namespace sr
