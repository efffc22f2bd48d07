// geom.cu — transform, count pass and fused intersect+fragment kernels.
//
// transform_pos.comp          -> k_transform
// make_intersection_0.comp    -> k_count
// make_intersection_1.comp    -> k_chains (the crossings), k_order_records
//                                (their order), k_merge (for a read-back)
// gen_fragment.comp           -> k_fragment
#include <algorithm>

#include "kernels.h"
#include "scan.cuh"
#include "segtiles.cuh"

namespace sr {

// ---------------------------------------------------------------- K1 ----
// transform_pos.comp:33-86.  One thread per point; the region-code OR into
// path_visible is aggregated over runs of equal path within a warp (points
// are grouped by path) before one atomicOr per run.  Beside that it clears the
// `zero` words, which only kernels after the offset scan use (a clear between
// that and the chains would be one more launch between two kernels).
__global__ void __launch_bounds__(256) k_transform(const float2* __restrict__ pos,
                                                   const uint32_t* __restrict__ pos_path, uint32_t n_points,
                                                   const SceneTable t, float2* __restrict__ tpos,
                                                   int32_t* __restrict__ path_visible, uint4* __restrict__ zero,
                                                   size_t zero_words) {
    wait_for_stream();
    for (size_t w = (size_t)blockIdx.x * blockDim.x + threadIdx.x; w < zero_words; w += (size_t)gridDim.x * blockDim.x)
        zero[w] = make_uint4(0u, 0u, 0u, 0u);
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t lane = lane_id();
    uint32_t pidx = 0xFFFFFFFFu;
    int32_t v = 0;
    if (i < n_points) {
        float2 p = pos[i];
        pidx = pos_path[i];
        const SceneInfo& si = scene_of_path(t, pidx);
        const float fw = (float)si.W, fh = (float)si.H;
        float o[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            // dot((x, y, 0, 1), m_r) summed left to right
            float acc = __fmul_rn(p.x, si.mvp[4 * r + 0]);
            acc = __fadd_rn(acc, __fmul_rn(p.y, si.mvp[4 * r + 1]));
            acc = __fadd_rn(acc, __fmul_rn(0.0f, si.mvp[4 * r + 2]));
            acc = __fadd_rn(acc, __fmul_rn(1.0f, si.mvp[4 * r + 3]));
            o[r] = acc;
        }
        float ox = __fdiv_rn(o[0], o[3]);
        float oy = __fdiv_rn(o[1], o[3]);
        tpos[i] = make_float2(ox, oy);
        int xf = ox < 0.0f ? 0 : (ox < fw ? 1 : 2);
        int yf = oy < 0.0f ? 0 : (oy < fh ? 1 : 2);
        switch ((yf << 4) | xf) {
            case 0x00: v = 0x10000000; break;
            case 0x01: v = 0x01000000; break;
            case 0x02: v = 0x00100000; break;
            case 0x10: v = 0x00010000; break;
            case 0x11: v = 0x10000001; break;
            case 0x12: v = 0x00001000; break;
            case 0x20: v = 0x00000100; break;
            case 0x21: v = 0x00000010; break;
            case 0x22: v = 0x00000001; break;
            default: break;
        }
    }
    // segmented OR-scan over runs of equal pidx
#pragma unroll
    for (uint32_t d = 1; d < 32; d <<= 1) {
        int32_t tv = __shfl_up_sync(0xFFFFFFFFu, v, d);
        uint32_t tp = __shfl_up_sync(0xFFFFFFFFu, pidx, d);
        if (lane >= d && tp == pidx) v |= tv;
    }
    uint32_t next = __shfl_down_sync(0xFFFFFFFFu, pidx, 1);
    bool run_end = (lane == 31) || (next != pidx);
    if (i < n_points && run_end && v != 0) atomicOr(&path_visible[pidx], v);
}

// Arcs, after k_transform (which took every slot for a point): the control
// slot (w*x, w*y) transforms linearly as (w*x, w*y, 0, w), the same dot
// products in the same order, with no division; the weight slot becomes the
// fourth row's result.  An arc with w <= 0 can leave the hull of its slots,
// so the region codes cannot cull it: its path is marked visible outright.
__global__ void __launch_bounds__(256) k_arc_fixup(const uint32_t* __restrict__ curve_type,
                                                   const uint32_t* __restrict__ curve_pos,
                                                   const uint32_t* __restrict__ curve_path, uint32_t n_curves,
                                                   const float2* __restrict__ pos, const SceneTable t,
                                                   float2* __restrict__ tpos, int32_t* __restrict__ path_visible) {
    wait_for_stream();
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n_curves || curve_type[c] != kArc) return;
    const uint32_t first = curve_pos[c], path = curve_path[c];
    const SceneInfo& si = scene_of_path(t, path);
    const float2 h = pos[first + 1];
    const float w = pos[first + 3].x;
    float o[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        float acc = __fmul_rn(h.x, si.mvp[4 * r + 0]);
        acc = __fadd_rn(acc, __fmul_rn(h.y, si.mvp[4 * r + 1]));
        acc = __fadd_rn(acc, __fmul_rn(0.0f, si.mvp[4 * r + 2]));
        acc = __fadd_rn(acc, __fmul_rn(w, si.mvp[4 * r + 3]));
        o[r] = acc;
    }
    tpos[first + 1] = make_float2(o[0], o[1]);
    tpos[first + 3] = make_float2(o[3], o[3]);
    atomicOr(&path_visible[path], 0x11111111);
}

// ------------------------------------------------- shared curve helpers --
struct CurvePts {
    float x[4], y[4];
};

SR_DEV void load_curve(const float2* __restrict__ tpos, uint32_t first, uint32_t type, CurvePts& c) {
    uint32_t np = curve_slots(type);
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
        float2 p = make_float2(0.0f, 0.0f);
        if (k < np) p = tpos[first + k];
        c.x[k] = p.x;
        c.y[k] = p.y;
    }
}

// interp() without a branch per curve type (but arcs): every level's lerps,
// and the level that the type ends at.  Warps hold mixed types.
SR_DEV float curve_coord(uint32_t type, float t, const float* p) {
    if (type == kArc) return interp(type, t, p);
    const float q0 = lerp_rn(p[0], p[1], t), q1 = lerp_rn(p[1], p[2], t), q2 = lerp_rn(p[2], p[3], t);
    const float l0 = lerp_rn(q0, q1, t), l1 = lerp_rn(q1, q2, t);
    const float b = lerp_rn(l0, l1, t);
    return type == 2u ? q0 : (type == 3u ? l0 : b);
}

// solveQuadEquation (make_intersection_0.comp:76-129)
SR_DEV void solve_quad(float a, float b, float c, float& r0, float& r1) {
    if (a == 0.0f) {
        float x = __fdiv_rn(-c, b);
        r0 = x;
        r1 = x;
        return;
    }
    float A = a, B = __fmul_rn(b, 0.5f), C = c;
    float R = __fsub_rn(__fmul_rn(B, B), __fmul_rn(A, C));
    if (R > 0.0f) {
        float SR = __fsqrt_rn(R);
        if (B > 0.0f) {
            float TB = __fadd_rn(B, SR);
            r0 = __fdiv_rn(-C, TB);
            r1 = __fdiv_rn(-TB, A);
        } else {
            float TB = __fadd_rn(-B, SR);
            r0 = __fdiv_rn(TB, A);
            r1 = __fdiv_rn(C, TB);
        }
    } else {
        r0 = 0.0f;
        r1 = 0.0f;
    }
}

// udpate_cut_range for one axis (make_intersection_0.comp:186-221)
SR_DEV int32_t cut_range(int32_t size, int32_t F, int32_t& b, int32_t& e) {
    int32_t mn = 0, mx = wadd(size & (int32_t)0xFFFFFFFE, F);
    if ((b < mn && e < mn) || (b > mx && e > mx) || (b > e)) return 0;
    b = iclamp(b, mn, mx);
    e = iclamp(e, mn, mx);
    return imax((e - b) / F + 1, 0);
}


// Pieces of a curve: at most 4 monotonic cuts + the end at t = 1.
constexpr int kMaxPieces = 5;
// A lane of a split chain takes at least 1 << kSegLog bisected roots: 64 when
// the chains are many waves of work (longer stretches waste fewer run-up and
// repeated roots), 8 when they leave schedulers idle (a lane's stretch is its
// latency).  "Many" and "few" by the warps' shares (tickets) that stretches of
// 16 would give.  The chain stage in ms, with 8 / 16 / 32 / 64: 4096^2 frame
// of 20,000 paths (45,000 tickets) 0.36 / 0.293 / 0.276 / 0.267, batch of 64
// uneven scenes 0.26 / 0.212 / 0.205 / 0.192, 2048^2 frame of 5,000 paths
// (10,291) 0.135 / 0.121 / 0.133, 1000x750 frame of 1,200 paths (1,906) 0.036 /
// 0.041, 1024^2 frame of 500 paths (1,001) 0.041 / 0.045 (4: 0.037).  (One
// chain a lane, and the longest a warp each beside them, took 1.35, 0.82 and
// 0.33 ms for the 4096^2, 2048^2 and 1024^2 frames.)
constexpr int32_t kSegShort = 3, kSegLog = 4, kSegLong = 6;
constexpr uint32_t kShortTickets = 16, kLongTickets = 160;   // an SM
constexpr int kChainCtas = 7;   // of four warps, an SM: all that fit with 72 registers a thread

// Piece record layout in the output: [t0][x crossings][y crossings], the
// crossing values of each side solved by one chain (k_chains), then merged
// in t order (k_merge).  PieceInfo packs what the chains and the merge need.
SR_DEV uint32_t pack_n(int32_t nx, bool xneg, int32_t ny, bool yneg) {
    return (uint32_t)nx | (xneg ? 0x8000u : 0u) | ((uint32_t)ny << 16) | (yneg ? 0x80000000u : 0u);
}
SR_DEV int32_t piece_nx(uint32_t n) { return (int32_t)(n & 0x7FFFu); }
SR_DEV int32_t piece_ny(uint32_t n) { return (int32_t)((n >> 16) & 0x7FFFu); }

// Class of a chain: longest length class first (so the longest chains start
// in the first wave of k_chains), then cubic, quadric, line, arc, so that a
// warp runs one curve type with lengths within a factor of 2.
constexpr uint32_t kChainClasses = 64;
constexpr uint32_t kEmptyPiece = 63;   // a piece without crossings: nothing to solve, one record
SR_DEV uint32_t chain_key(int32_t len, uint32_t type) {
    uint32_t lg = 31u - (uint32_t)__clz(len);
    if (lg > 14u) lg = 14u;
    uint32_t cls = type == 4u ? 0u : (type == 3u ? 1u : (type == kArc ? 3u : 2u));
    return ((14u - lg) << 2) | cls;
}
// How the chains of a class are shared out: 2^lanes lanes a chain and 2^warps
// warps (warps only with 32 lanes).  Solving, a lane takes 1 << seg_log to
// twice that bisected roots or, a line's root being a closed form, 32 times as
// many of a line, as far as 32 lanes go (run_segments).  Ordering, a lane takes every 32nd root, up
// to 256 a warp, so that a warp's roots are neighbours in memory.
struct ChainShare {
    uint32_t lanes, warps;
};
template <bool kSolve> SR_DEV ChainShare chain_share(uint32_t key, int32_t seg_log) {
    const int32_t lg = 14 - (int32_t)(key >> 2);
    ChainShare s;
    s.lanes = (uint32_t)imin(imax(kSolve ? lg - ((key & 3u) == 2u ? seg_log + 5 : seg_log) : lg + 1, 0), 5);
    s.warps = kSolve ? 0u : (uint32_t)imax(lg + 1 - 8, 0);
    return s;
}

// get_xy_begin_end_delta + udpate_cut_range for one axis
// (make_intersection_1.comp:150-213): number of grid crossings, first
// grid line and step.
SR_DEV int32_t axis_range_rd(float a0, float a1, int32_t size, int32_t F, float& start, bool& neg) {
    const float invF = inv_F(F);   // x / F == x * (1/F) exactly for F in {1, 2}
    int32_t b, e;
    if (a0 <= a1) {
        b = wadd(wmul(float2int_rd(__fmul_rn(a0, invF)), F), F);
        e = wmul(float2int_rd(__fmul_rn(a1, invF)), F);
        neg = false;
    } else {
        b = wadd(wmul(float2int_rd(__fmul_rn(a1, invF)), F), F);
        e = wmul(float2int_rd(__fmul_rn(a0, invF)), F);
        neg = true;
    }
    int32_t n = cut_range(size, F, b, e);
    start = (float)(neg ? e : b);
    return n;
}

// out[from, to) = value, by the CTA.
SR_DEV void fill_range(uint32_t* __restrict__ out, uint32_t from, uint32_t to, uint32_t value) {
    const uint32_t t = threadIdx.x, nt = blockDim.x;
    const uint32_t a = min((from + 3u) & ~3u, to), b = max(to & ~3u, a);   // whole 16 bytes between
    if (from + t < a) out[from + t] = value;
    for (uint32_t q = a + 4 * t; q < b; q += 4 * nt)
        *reinterpret_cast<uint4*>(out + q) = make_uint4(value, value, value, value);
    if (b + t < to) out[b + t] = value;
}

// ---------------------------------------------------------------- K2 ----
// Paths without curves in a row that a curve's own thread gives their first
// curve; longer rows take its CTA (2 million such paths took a thread alone 9
// ms, a warp 0.17, the CTA 0.12).
constexpr uint32_t kPathGap = 32;
// LANES 8: eight lanes a curve, a piece each, for a frame of few curves, whose
// time is one curve's serial set-up: 9.8 instead of 15 us for 5,000 curves (but
// 23 instead of 19 for 60,000, where the lanes' repeated cuts count).
constexpr uint32_t kFewCurves = 16384;
constexpr int kCountThreads = 128;   // 256: 0.043 instead of 0.039 ms for 200,000 curves
// make_intersection_0.comp:226-411.  One thread per curve: path cull,
// monotonic cut points (cached, 5 floats per curve), the number of records
// the curve emits (the reference's count), and the set-up of each piece's
// x and y crossing chains, which are appended with their sort keys.
template <int LANES>
__global__ void __launch_bounds__(kCountThreads) k_count(const GeomArgs g, float* __restrict__ cut_cache,
                                               int32_t* __restrict__ count, uint4* __restrict__ pieces,
                                               uint32_t* __restrict__ chain_items, uint8_t* __restrict__ chain_keys,
                                               uint32_t list_cap, uint32_t* __restrict__ chain_count,
                                               uint32_t* __restrict__ class_count, uint32_t* __restrict__ status) {
    wait_for_stream();
    __shared__ uint32_t s_hist[kChainClasses], s_total, s_base;
    __shared__ uint3 s_gap[kCountThreads / LANES + 1];   // paths [x, y) begin at curve z
    __shared__ uint32_t s_gaps;
    const uint32_t c = (blockIdx.x * blockDim.x + threadIdx.x) / LANES;
    const uint32_t sub = LANES == 1 ? 0u : threadIdx.x % LANES;   // the piece that this lane sets up
    const bool active = c < g.n_curves;
    if (threadIdx.x < kChainClasses) s_hist[threadIdx.x] = 0;
    if (threadIdx.x == kChainClasses) s_total = s_gaps = 0;
    __syncthreads();
    constexpr int kMine = LANES == 1 ? kMaxPieces : 1;   // pieces a lane
    uint32_t my_chains[2 * kMine];
    uint32_t my_key[2 * kMine];
    int32_t pc = 0, walk = 0;
    int n_chains = 0;
    if (active) {
        uint32_t type = g.curve_type[c];
        CurvePts P;
        load_curve(g.tpos, g.curve_pos[c], type, P);
        const uint32_t path = g.curve_path[c];
        bool vis = path_visible_mask(g.path_visible[path]);
        const SceneInfo& si = scene_of_path(g.st, path);
        const int32_t W = si.W, H = si.H;
        const int32_t F = g.F;
        uint32_t n = 0;
        float q[5] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        if (vis) {
#pragma unroll
            for (int ax = 0; ax < 2; ++ax) {
                const float* p = ax == 0 ? P.x : P.y;
                if (type == 4u) {
                    float r0 = 0.0f, r1 = 0.0f;
                    float a = __fadd_rn(__fmul_rn(3.0f, __fsub_rn(p[1], p[2])), __fsub_rn(p[3], p[0]));
                    float b = __fmul_rn(2.0f, __fadd_rn(__fsub_rn(p[0], p[1]), __fsub_rn(p[2], p[1])));
                    solve_quad(a, b, __fsub_rn(p[1], p[0]), r0, r1);
                    if (r0 > 0.0f && r0 < 1.0f) q[n++] = r0;
                    if (r1 > 0.0f && r1 < 1.0f && r1 != r0) q[n++] = r1;
                } else if (type == 3u) {
                    float den = __fadd_rn(__fsub_rn(p[0], p[1]), __fsub_rn(p[2], p[1]));
                    if (den != 0.0f) {
                        float r0 = __fdiv_rn(__fsub_rn(p[0], p[1]), den);
                        if (r0 > 0.0f && r0 < 1.0f) q[n++] = r0;
                    }
                } else if (type == kArc) {
                    // roots of the derivative's numerator N'D - ND' (a
                    // quadratic; its cubic terms cancel), halved:
                    // (w-1)(x2-x0) t^2 + ((x0-x1) + (x2-x1) + 2 x0 (w-1)) t + (x1 - w x0)
                    const float wm1 = __fsub_rn(p[3], 1.0f);
                    float r0 = 0.0f, r1 = 0.0f;
                    solve_quad(__fmul_rn(wm1, __fsub_rn(p[2], p[0])),
                               __fadd_rn(__fadd_rn(__fsub_rn(p[0], p[1]), __fsub_rn(p[2], p[1])),
                                         __fmul_rn(__fmul_rn(2.0f, p[0]), wm1)),
                               __fsub_rn(p[1], __fmul_rn(p[3], p[0])), r0, r1);
                    if (r0 > 0.0f && r0 < 1.0f) q[n++] = r0;
                    if (r1 > 0.0f && r1 < 1.0f && r1 != r0) q[n++] = r1;
                }
            }
            // insertion network of make_intersection_0.comp:315-359, including
            // its `t2 = q3` (the 4th cut is never moved)
            float q0 = q[0], q1 = q[1], q2 = q[2], q3 = q[3];
            if (n >= 2) {
                float t1 = q1, t0 = q0;
                if (t1 < t0) { q1 = t0; q0 = t1; }
            }
            if (n >= 3) {
                float t2 = q2, t1 = q1;
                if (t2 < t1) {
                    q2 = t1;
                    float t0 = q0;
                    if (t2 < t0) { q1 = t0; q0 = t2; } else { q1 = t2; }
                }
            }
            if (n >= 4) {
                float t3 = q3, t2 = q3;
                if (t3 < t2) {
                    q3 = t2;
                    float t1 = q1;
                    if (t3 < t1) {
                        q2 = t1;
                        float t0 = q0;
                        if (t3 < t0) { q1 = t0; q0 = t3; } else { q1 = t3; }
                    } else {
                        q2 = t3;
                    }
                }
            }
            q[0] = q0; q[1] = q1; q[2] = q2; q[3] = q3;
        }
        if (sub == 0) {
            float* cc = cut_cache + 5 * (size_t)c;
            cc[0] = q[0];
            cc[1] = q[1];
            cc[2] = q[2];
            cc[3] = q[3];
            cc[4] = __uint_as_float(n);
        }
        if (vis) q[n++] = 1.0f;
        float x0 = P.x[0], y0 = P.y[0];
        const float fF = (float)F, inv = inv_F(F);   // x / F == x * (1/F) exactly
        uint4* pt = pieces + (size_t)c * kMaxPieces;
        float t_mine = 0.0f;
        if (LANES > 1) {   // this lane's piece starts where the one before it ends
            float t_from = 0.0f;
#pragma unroll
            for (int k = 0; k < kMaxPieces; ++k) {
                if ((uint32_t)k + 1u == sub) t_from = q[k];
                if ((uint32_t)k == sub) t_mine = q[k];
            }
            if (sub > 0 && sub < n) {
                x0 = curve_coord(type, t_from, P.x);
                y0 = curve_coord(type, t_from, P.y);
            }
        }
#pragma unroll
        for (uint32_t j = 0; j < (uint32_t)kMine; ++j) {
            const uint32_t i = LANES == 1 ? j : sub;
            if (i >= n) break;
            float t1 = LANES == 1 ? q[j] : t_mine;
            float x1 = curve_coord(type, t1, P.x), y1 = curve_coord(type, t1, P.y);
            // count: get_xy_begin_end (make_intersection_0.comp:167-183)
            int32_t xb, xe, yb, ye;
            if (x0 <= x1) {
                xb = wadd(f2i(__fmul_rn(floorf(__fmul_rn(x0, inv)), fF)), F);
                xe = f2i(__fmul_rn(floorf(__fmul_rn(x1, inv)), fF));
            } else {
                xb = wadd(f2i(__fmul_rn(floorf(__fmul_rn(x1, inv)), fF)), F);
                xe = f2i(__fmul_rn(floorf(__fmul_rn(x0, inv)), fF));
            }
            if (y0 <= y1) {
                yb = wadd(f2i(__fmul_rn(floorf(__fmul_rn(y0, inv)), fF)), F);
                ye = f2i(__fmul_rn(floorf(__fmul_rn(y1, inv)), fF));
            } else {
                yb = wadd(f2i(__fmul_rn(floorf(__fmul_rn(y1, inv)), fF)), F);
                ye = f2i(__fmul_rn(floorf(__fmul_rn(y0, inv)), fF));
            }
            int32_t nxc = cut_range(W, F, xb, xe);
            int32_t nyc = cut_range(H, F, yb, ye);
            pc = wadd(pc, wadd(1, wadd(nxc, nyc)));
            // chain set-up: the intersection pass's own range formulas
            float sx, sy;
            bool xneg, yneg;
            int32_t nx = axis_range_rd(x0, x1, W, F, sx, xneg);
            int32_t ny = axis_range_rd(y0, y1, H, F, sy, yneg);
            int32_t tb = fbits(t1) & ~3;
            tb |= (floorf(x1) == x1) ? 2 : 3;   // make_intersection_1.comp:271-276
            pt[i] = make_uint4(pack_n(nx, xneg, ny, yneg), (uint32_t)tb, __float_as_uint(sx), __float_as_uint(sy));
            if (nx > 0) {
                my_chains[n_chains] = (c << 4) | (i << 1) | 0u;
                my_key[n_chains++] = chain_key(nx, type);
            }
            if (ny > 0) {
                my_chains[n_chains] = (c << 4) | (i << 1) | 1u;
                my_key[n_chains++] = chain_key(ny, type);
            }
            if (nx <= 0 && ny <= 0) {   // a record of its own start only
                my_chains[n_chains] = (c << 4) | (i << 1);
                my_key[n_chains++] = kEmptyPiece;
            }
            walk += 1 + nx + ny;
            x0 = x1;
            y0 = y1;
        }
        // the point at t = 1 (without pieces, the start)
        if (LANES == 1 || sub + 1u == n || (n == 0 && sub == 0)) g.curve_end[c] = make_float2(x0, y0);
    }
    if (LANES > 1) {   // the curve's sums, in its first lane
#pragma unroll
        for (int d = LANES / 2; d; d >>= 1) {
            pc = wadd(pc, __shfl_down_sync(0xFFFFFFFFu, pc, d, LANES));
            walk = wadd(walk, __shfl_down_sync(0xFFFFFFFFu, walk, d, LANES));
        }
    }
    if (active && sub == 0) {
        const uint32_t path = g.curve_path[c];
        count[c] = pc;
        // first curve of every path up to this curve's (curves are grouped by
        // path, in order; a path without curves starts where the next does)
        const uint32_t first = c ? g.curve_path[c - 1] + 1u : 0u;
        if (path + 1u - first > kPathGap) {
            s_gap[atomicAdd(&s_gaps, 1u)] = make_uint3(first, path + 1u, c);
        } else {
            for (uint32_t q = first; q <= path; ++q) g.path_begin[q] = c;
        }
        if (c == g.n_curves - 1) s_gap[atomicAdd(&s_gaps, 1u)] = make_uint3(path + 1u, g.n_paths + 1u, g.n_curves);
        if (walk != pc) set_error(status, ERR_RECORD_RANGE);
    }
    // append the chains with their classes, and count the classes (one
    // append and at most one add per class for the CTA)
    uint32_t at = 0;
    if (n_chains) at = atomicAdd(&s_total, (uint32_t)n_chains);
    for (int k = 0; k < n_chains; ++k) atomicAdd(&s_hist[my_key[k]], 1u);
    __syncthreads();
    for (uint32_t i = 0; i < s_gaps; ++i) fill_range(g.path_begin, s_gap[i].x, s_gap[i].y, s_gap[i].z);
    if (threadIdx.x < kChainClasses && s_hist[threadIdx.x]) atomicAdd(&class_count[threadIdx.x], s_hist[threadIdx.x]);
    if (threadIdx.x == kChainClasses && s_total) s_base = atomicAdd(chain_count, s_total);
    __syncthreads();
    for (int k = 0; k < n_chains; ++k) {
        const uint32_t slot = s_base + at + (uint32_t)k;
        if (slot < list_cap) {
            chain_items[slot] = my_chains[k];
            chain_keys[slot] = (uint8_t)my_key[k];
        } else {
            set_error(status, ERR_CAPACITY);
        }
    }
}

// First list position of each class: an exclusive scan of the class counts
// by one warp (two classes a lane).
SR_DEV void class_starts(const uint32_t* __restrict__ class_count, uint32_t& s0, uint32_t& s1) {
    const uint32_t lane = lane_id();
    const uint32_t a = class_count[2 * lane], b = class_count[2 * lane + 1];
    uint32_t x = a + b;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, d);
        if ((int)lane >= d) x += y;
    }
    s0 = x - a - b;
    s1 = s0 + a;
}

// Two things that follow the count pass and do not touch each other, in one
// launch (a launch costs 2-3 us of a small frame): the first scan_tiles CTAs
// scan the curves' counts into their record offsets; the others order the
// chains by class (in no order within one), a counting sort whose counts the
// count pass made (the radix sort that it replaced took five launches).  The
// scan's last tile also leaves the record count in report_n.
constexpr int kOffsetRows = 1;   // small tiles: 240 K curves are 234 of them
// (a curve gives at most kMaxPieces * (1 + 2 * 16,387) records)
static_assert(1024ull * kOffsetRows * kMaxPieces * (1 + 2 * 16387) < (1ull << 28), "records a tile adds");
__global__ void __launch_bounds__(256) k_offsets_and_order(
    const int32_t* __restrict__ count, int32_t* __restrict__ offs, uint32_t n_curves, uint32_t scan_tiles,
    uint64_t* tstat, uint32_t* counter, uint32_t* report_n, uint32_t* status, uint32_t spin_limit,
    const uint32_t* __restrict__ items, const uint8_t* __restrict__ keys, uint32_t list_cap,
    const uint32_t* __restrict__ chain_count, const uint32_t* __restrict__ class_count,
    uint32_t* __restrict__ class_next, uint32_t* __restrict__ sorted) {
    wait_for_stream();
    __shared__ uint32_t s_start[kChainClasses], s_hist[kChainClasses], s_at[kChainClasses];
    __shared__ uint32_t s_tile;
    __shared__ int32_t s_warp[256 / 32 + 1];
    if (blockIdx.x < scan_tiles) {
        if (threadIdx.x == 0) s_tile = atomicAdd(counter, 1u);
        __syncthreads();
        int32_t total;
        const bool last =
            scan_tile_i32<kOffsetRows, 256>(count, offs, n_curves, s_tile, tstat, status, spin_limit, s_warp, &total);
        if (threadIdx.x == 0) {
            if (last) *report_n = (uint32_t)total;
            // More records than a frame takes, whatever the sum has become by
            // the end: a tile adds less than 2^28, so no sum passes 2^31
            // without a tile that ends between 2^30 and there.
            if ((uint32_t)total >= kMaxRecords) set_error(status, ERR_CAPACITY);
        }
        return;
    }
    const uint32_t n = imin((int32_t)*chain_count, (int32_t)list_cap);
    if (threadIdx.x < 32) {
        uint32_t a, b;
        class_starts(class_count, a, b);
        s_start[2 * threadIdx.x] = a;
        s_start[2 * threadIdx.x + 1] = b;
    }
    for (uint32_t i0 = (blockIdx.x - scan_tiles) * 256u; i0 < n; i0 += (gridDim.x - scan_tiles) * 256u) {
        if (threadIdx.x < kChainClasses) s_hist[threadIdx.x] = 0;
        __syncthreads();
        const uint32_t i = i0 + threadIdx.x;
        uint32_t key = 0, rank = 0;
        if (i < n) {
            key = keys[i];
            rank = atomicAdd(&s_hist[key], 1u);
        }
        __syncthreads();
        if (threadIdx.x < kChainClasses && s_hist[threadIdx.x])
            s_at[threadIdx.x] = s_start[threadIdx.x] + atomicAdd(&class_next[threadIdx.x], s_hist[threadIdx.x]);
        __syncthreads();
        if (i < n) {
            const uint32_t o = s_at[key] + rank;
            if (o < list_cap) sorted[o] = items[i];
        }
    }
}

// ------------------------------------------------------------ chains -----
// One crossing chain: the successive roots of one coordinate of one piece
// at the grid lines start, start+d, ... (make_intersection_1.comp:377-440).
// Each solve starts from the previous root of the same side (flag bits
// included), so a chain is sequential but chains are independent.
struct AxisPoly {
    float p0, p1, p2, p3;
    float d01, d12, d23;
};

template <int kType> SR_DEV float eval_axis(const AxisPoly& a, float t) {
    if (kType == 2) return __fadd_rn(a.p0, __fmul_rn(t, a.d01));
    if (kType == (int)kArc) {
        // as interp(): the homogeneous lerps, then the division (p3 = w)
        float q0 = __fadd_rn(a.p0, __fmul_rn(t, a.d01));
        float q1 = __fadd_rn(a.p1, __fmul_rn(t, a.d12));
        float r0 = __fadd_rn(1.0f, __fmul_rn(t, __fsub_rn(a.p3, 1.0f)));
        float r1 = __fadd_rn(a.p3, __fmul_rn(t, __fsub_rn(1.0f, a.p3)));
        return __fdiv_rn(__fadd_rn(q0, __fmul_rn(t, __fsub_rn(q1, q0))),
                         __fadd_rn(r0, __fmul_rn(t, __fsub_rn(r1, r0))));
    }
    float q0 = __fadd_rn(a.p0, __fmul_rn(t, a.d01));
    float q1 = __fadd_rn(a.p1, __fmul_rn(t, a.d12));
    if (kType == 3) return __fadd_rn(q0, __fmul_rn(t, __fsub_rn(q1, q0)));
    float q2 = __fadd_rn(a.p2, __fmul_rn(t, a.d23));
    float l0 = __fadd_rn(q0, __fmul_rn(t, __fsub_rn(q1, q0)));
    float l1 = __fadd_rn(q1, __fmul_rn(t, __fsub_rn(q2, q1)));
    return __fadd_rn(l0, __fmul_rn(t, __fsub_rn(l1, l0)));
}

SR_DEV float mid_rn(float lo, float hi) { return __fmul_rn(__fadd_rn(lo, hi), 0.5f); }

// The step test of make_intersection_1.comp:421 is
// (bits(v - c) ^ bits(v_lo - c)) >= 0, v_lo the value at the interval's low
// end; for finite values v - c is negative exactly when v < c (x - x is +0).
// The low end moves only to a midpoint that passes the test, i.e. one on the
// same side of c, so the side s0 = (value at t_min < c) holds for the whole
// solve: a step goes right exactly when (v < c) == s0, whatever the other
// steps did.  Both solvers below rest on that.

// 24-step bisection of the reference (make_intersection_1.comp:402-434), a
// thread per chain.  (Evaluating both possible next midpoints with each one
// halves the dependent depth, but the chains left to this solver are
// throughput-bound, and the extra evaluations made the frame slower.)
template <int kType>
SR_DEV float bisect(const AxisPoly& a, float c, float t_min, float t_max) {
    const float v0 = eval_axis<kType>(a, t_min);
    const bool s0 = v0 < c;
    float ta = t_min, tb = t_max;
    float t_solve = t_min, last = 0.0f;
#pragma unroll 4
    for (int j = 0; j < 24; ++j) {
        const float tm = mid_rn(ta, tb);
        const float v = eval_axis<kType>(a, tm);
        t_solve = tm;
        last = v;
        if ((v < c) == s0) ta = tm;
        else tb = tm;
    }
    // vt0 == c returns t_min at once; a solve that ends more than one unit
    // away from c falls back to t_min too
    if (v0 == c || fabsf(__fsub_rn(last, c)) > 1.0f) t_solve = t_min;
    return t_solve;
}

// The same solve near a guess of its result: the turns of the first kGuessed
// steps are taken from the guess at once, so the midpoints do not wait for the
// values, and the values, which then depend on nothing but their midpoints,
// say whether every turn was right.  If one was not (a guess that is not the
// result's neighbour), the solve is done plainly.  1,150 cycles a root where
// the plain one takes 1,560: the chain stage of the 1024^2 frame went from
// 0.050 to 0.043 ms, of the 2048^2 one from 0.140 to 0.124 (14 turns: 0.045
// and 0.127; 20: no better).
constexpr int kGuessed = 18;
template <int kType>
SR_DEV float bisect_near(const AxisPoly& a, float c, float t_min, float t_max, float guess) {
    const float v0 = eval_axis<kType>(a, t_min);
    const bool s0 = v0 < c;
    float ta = t_min, tb = t_max;
    bool wrong = false;
#pragma unroll
    for (int j = 0; j < kGuessed; ++j) {
        const float tm = mid_rn(ta, tb);
        const bool right = tm < guess;
        if (right) ta = tm;
        else tb = tm;
        wrong |= ((eval_axis<kType>(a, tm) < c) == s0) != right;
    }
    if (wrong) return bisect<kType>(a, c, t_min, t_max);
    float t_solve = t_min, last = 0.0f;
#pragma unroll
    for (int j = kGuessed; j < 24; ++j) {
        const float tm = mid_rn(ta, tb);
        const float v = eval_axis<kType>(a, tm);
        t_solve = tm;
        last = v;
        if ((v < c) == s0) ta = tm;
        else tb = tm;
    }
    if (v0 == c || fabsf(__fsub_rn(last, c)) > 1.0f) t_solve = t_min;
    return t_solve;
}

// The state after root k of a chain whose state before it is lo: its t with
// the side bit in the flag bits.
struct ChainSide {
    AxisPoly a;
    float inv;            // 1 / (p1 - p0) of a line
    float x, dx, t_hi;    // first grid line, step, end of the piece
    int side;
};
//
// A line's root is NaN where the line starts on the grid line and is so short
// that 1 / (p1 - p0) overflows (0 * inf; it crosses no second line then), and
// all its roots are where the matrix sent a point to infinity.  No comparison
// holds for NaN, so the sequential merge never takes an x root that is one: t0
// and the y roots go before, and the exhausted y side's 2.0 stands in its
// place.  A y root that is NaN it takes at once, before any x root above t0.
// Stored as 2.0 and as -inf the two have these places in the order of numbers
// (k_order_records and k_merge write NaN for -inf).
constexpr int32_t kPastEnd = 0x40000001;            // 2.0 with the y side's bit
constexpr int32_t kNanY = (int32_t)0xFF800000u;     // -inf
SR_DEV int32_t stored_t(int32_t root) { return root == kNanY ? 0x7FFFFFFD : root; }
template <int kType> SR_DEV int32_t next_root(const ChainSide& s, int32_t k, int32_t lo) {
    // x + k dx: whole numbers below 2^15, exact like the repeated sum
    const float c = __fadd_rn(s.x, __fmul_rn((float)k, s.dx));
    float t;
    if (kType == 2) {
        t = gmin(gmax(__fmul_rn(__fsub_rn(c, s.a.p0), s.inv), bitsf(lo)), s.t_hi);
        if (t != t) return s.side ? kNanY : kPastEnd;
    } else {
        t = bisect<kType>(s.a, c, bitsf(lo), s.t_hi);
    }
    return (fbits(t) & ~3) | s.side;
}

// The same for a root whose state is likely near `guess`.
template <int kType> SR_DEV int32_t next_root_near(const ChainSide& s, int32_t k, int32_t lo, int32_t guess) {
    if (kType == 2) return next_root<kType>(s, k, lo);
    const float c = __fadd_rn(s.x, __fmul_rn((float)k, s.dx));
    return (fbits(bisect_near<kType>(s.a, c, bitsf(lo), s.t_hi, bitsf(guess))) & ~3) | s.side;
}

// Warp-cooperative solve of one long chain.  By the invariant above, the 31
// midpoints of the next five bisection steps can be evaluated at once: lane
// l holds node l+1 of the complete binary tree of those steps in heap order
// (node n's children are 2n and 2n+1, the right child taken when the step
// goes right), and one ballot of the (v < c) bits gives every node's turn.
// The leaf whose ancestors all turn toward it is on the path; it hands the
// new interval to the warp through a max-reduction over the lanes (every
// other lane offers 0; t >= 0, so the bit patterns order like the values).  Lane 31 evaluates the root's t_min in the first
// round, which gives s0 in the same ballot.  24 steps = four 5-level rounds
// and a last 4-level round, whose leaf midpoint is the 24th midpoint.
struct TreeLane {
    int32_t depth;            // node depth (lane 31: -1)
    bool d1, d2, d3, d4;      // turn at level j toward this lane's node (right = true)
    uint32_t anc5, want5, anc4, want4;   // path masks of the leaves of a 5- and a 4-level round
};

SR_DEV TreeLane tree_lane(uint32_t lane) {
    TreeLane tl;
    const uint32_t n = lane + 1u;
    const int32_t d = lane == 31u ? -1 : 31 - __clz((int32_t)n);
    tl.depth = d;
    tl.d1 = d >= 1 && ((n >> (d - 1)) & 1u);
    tl.d2 = d >= 2 && ((n >> (d - 2)) & 1u);
    tl.d3 = d >= 3 && ((n >> (d - 3)) & 1u);
    tl.d4 = d >= 4 && (n & 1u);
    tl.anc5 = tl.want5 = tl.anc4 = tl.want4 = 0;
    for (int32_t i = 0; i < d; ++i) {   // ancestor at depth i and the turn it takes toward n
        const uint32_t anc = n >> (d - i), dir = (n >> (d - i - 1)) & 1u;
        const uint32_t bit = 1u << (anc - 1u);
        if (d == 4) { tl.anc5 |= bit; tl.want5 |= dir ? bit : 0u; }
        if (d == 3) { tl.anc4 |= bit; tl.want4 |= dir ? bit : 0u; }
    }
    return tl;
}

// This lane's node of a kLevels-level tree from [ta, tb]: its midpoint,
// and its interval in lb/rb.  m_j = (m_{j-1} + the interval's other end) *
// 0.5, the other end being older than m_{j-1}, so a level costs one add and
// one multiply on the dependency path.
template <int kLevels>
SR_DEV float tree_node(float ta, float tb, const TreeLane& tl, float& lb, float& rb) {
    lb = ta;
    rb = tb;
    float m = mid_rn(ta, tb);
#pragma unroll
    for (int j = 1; j < kLevels; ++j) {
        if (j <= tl.depth) {
            const bool dir = j == 1 ? tl.d1 : (j == 2 ? tl.d2 : (j == 3 ? tl.d3 : tl.d4));
            const float other = dir ? rb : lb;
            if (dir) lb = m;
            else rb = m;
            m = __fmul_rn(__fadd_rn(m, other), 0.5f);
        }
    }
    return m;
}

template <int kType>
SR_DEV float bisect_warp(const AxisPoly& a, float c, float t_min, float t_max, const TreeLane& tl) {
    float lb, rb;
    // first round; lane 31's interval is [t_min, t_min], whose midpoint is
    // t_min itself (2t and 2t * 0.5 are exact), so its bit of the ballot is s0
    float m = tree_node<5>(t_min, tl.depth < 0 ? t_min : t_max, tl, lb, rb);
    float v = eval_axis<kType>(a, m);
    uint32_t B = __ballot_sync(0xFFFFFFFFu, v < c);
    const bool s0 = (B >> 31) & 1u;
    const bool eq0 = (__ballot_sync(0xFFFFFFFFu, v == c) >> 31) != 0u;
    // node l+1 goes right when bit l of B equals s0: the leaf on the path is
    // the one with ((B ^ key) & anc) == 0, key = want ^ (s0 ? 0 : ~0)
    const uint32_t flip = s0 ? 0u : 0xFFFFFFFFu;
    const uint32_t key5 = tl.want5 ^ flip, key4 = tl.want4 ^ flip;
    float ta, tb;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        if (r > 0) {
            m = tree_node<5>(ta, tb, tl, lb, rb);
            v = eval_axis<kType>(a, m);
            B = __ballot_sync(0xFFFFFFFFu, v < c);
        }
        const bool on = tl.depth == 4 && ((B ^ key5) & tl.anc5) == 0u;
        const bool right = (v < c) == s0;
        const uint32_t nta = on ? __float_as_uint(right ? m : lb) : 0u;
        const uint32_t ntb = on ? __float_as_uint(right ? rb : m) : 0u;
        ta = __uint_as_float(__reduce_max_sync(0xFFFFFFFFu, nta));
        tb = __uint_as_float(__reduce_max_sync(0xFFFFFFFFu, ntb));
    }
    // steps 21-24: the chosen depth-3 node's midpoint is the 24th midpoint
    m = tree_node<4>(ta, tb, tl, lb, rb);
    v = eval_axis<kType>(a, m);
    B = __ballot_sync(0xFFFFFFFFu, v < c);
    const bool on = tl.depth == 3 && ((B ^ key4) & tl.anc4) == 0u;
    const float fin = fabsf(__fsub_rn(v, c)) > 1.0f ? t_min : m;
    const float t = __uint_as_float(__reduce_max_sync(0xFFFFFFFFu, on ? __float_as_uint(fin) : 0u));
    return eq0 ? t_min : t;
}

// The rest of run_segments for a chain of 32 lanes some of which disagree:
// the first stretch whose entry state is not its neighbour's end is solved
// root by root by the whole warp, until the state meets a root that is there
// already, and so on to the next.
template <int kType>
SR_DEV void finish_chain_warp(const ChainSide& s, int32_t len, int32_t seg, int32_t* __restrict__ out, int32_t entry,
                              int32_t end) {
    const int32_t lane = (int32_t)lane_id();
    const TreeLane tl = tree_lane((uint32_t)lane);
    for (;;) {
        const int32_t prev = __shfl_up_sync(0xFFFFFFFFu, end, 1);
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, lane > 0 && lane * seg < len && prev != entry);
        if (!m) return;
        const int32_t f = __ffs(m) - 1;
        int32_t st = __shfl_sync(0xFFFFFFFFu, prev, f);
        if (lane == f) entry = st;
        const int32_t k1 = imin((f + 1) * seg, len);
        bool met = false;
        for (int32_t k = f * seg; k < k1 && !met; ++k) {
            const float c = __fadd_rn(s.x, __fmul_rn((float)k, s.dx));
            const float t = bisect_warp<kType>(s.a, c, bitsf(st), s.t_hi, tl);
            st = (fbits(t) & ~3) | s.side;
            met = out[k] == st;
            __syncwarp();
            if (lane == 0) out[k] = st;
        }
        if (lane == f && !met) end = st;
        __syncwarp();
    }
}

// One chain by `lanes` lanes, lane l of them taking the roots [ks, ke) of
// its stretch.  A root depends on the one before it only through the low end
// of its interval, and by little: the 24 steps end within 2^-24 of the
// interval from the crossing wherever they start, and the state keeps t to
// 4 ulp.  So two chains started from different low ends soon hold the same
// state (on the generated scenes, after two roots in 95% of the cases; later
// for t under an eighth of the piece, where 4 ulp is finer than the steps'
// end).  Each lane starts a root before its stretch from the piece's own start
// and solves on from there (a second run-up root saves fewer repeats than it
// costs: 0.041 instead of 0.035 ms on the 1024^2 frame); then every lane whose state at its
// stretch's start is not the one its left neighbour ended with solves again
// from that one, near the roots it has (bisect_near), until it meets one of
// them.  Rounds of this end when all neighbours agree, which makes every root the one that the
// sequential chain gives.  A chain of 32 lanes that has not settled after a
// round (its t small all along) is finished root by root by the warp.
template <int kType>
SR_DEV void run_segments(const ChainSide& s, int32_t len, float t_lo, int32_t* __restrict__ out, int32_t lanes,
                         int32_t l) {
    const int32_t seg = (len + lanes - 1) / lanes;
    const int32_t ks = imin(l * seg, len), ke = imin(ks + seg, len);
    int32_t st = fbits(t_lo);
    if (ks < ke)
        for (int32_t k = imax(ks - 1, 0); k < ks; ++k) st = next_root<kType>(s, k, st);
    int32_t entry = st;
    for (int32_t k = ks; k < ke; ++k) {
        st = next_root<kType>(s, k, st);
        out[k] = st;
    }
    int32_t end = st;
    __syncwarp();
    for (int round = 0;; ++round) {
        const int32_t prev = __shfl_up_sync(0xFFFFFFFFu, end, 1);
        const bool need = l > 0 && ks < ke && prev != entry;
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, need);
        if (!m) return;
        if (kType != 2 && lanes == 32 && round >= 1) {
            finish_chain_warp<kType>(s, len, seg, out, entry, end);
            return;
        }
        if (need) {
            entry = prev;
            st = prev;
            bool met = false;
            for (int32_t k = ks; k < ke; ++k) {
                const int32_t was = out[k];   // solved from another low end: a neighbour of this one
                st = next_root_near<kType>(s, k, st, was);
                met = was == st;
                if (met) break;
                out[k] = st;
            }
            if (!met) end = st;
        }
        __syncwarp();
    }
}

constexpr uint32_t kBackwards = 0x8000u;   // a piece that runs backwards (its x crossings take 15 bits)

struct ChainSetup {
    uint4 piece;   // of the record order: first record, crossings (pack_n without signs, kBackwards), start bits, item
    ChainSide side;
    uint32_t type;
    int32_t len;
    float t_lo;
    int64_t base;
};

// Chain item (curve << 4 | piece << 1 | side): its polynomial, first grid
// line and step, t range and output slot.
SR_DEV ChainSetup chain_setup(const GeomArgs& g, const int32_t* __restrict__ offs, const uint4* __restrict__ pieces,
                              uint32_t item) {
    ChainSetup s;
    const uint32_t c = item >> 4, piece = (item >> 1) & 7u;
    const int side = (int)(item & 1u);
    s.side.side = side;
    s.type = g.curve_type[c];
    const uint4* pt = pieces + (size_t)c * kMaxPieces;
    int64_t base = offs[c];
    for (uint32_t j = 0; j < piece; ++j) base += 1 + piece_nx(pt[j].x) + piece_ny(pt[j].x);
    const uint4 me = pt[piece];
    const int32_t nx = piece_nx(me.x), ny = piece_ny(me.x);
    s.base = base + 1 + (side ? nx : 0);
    s.len = side ? ny : nx;
    const uint32_t t0 = piece == 0 ? 0u : pt[piece - 1].y;   // bits of 0.0f for the first piece
    const bool back = __uint_as_float(me.y) < __uint_as_float(t0);
    s.piece = make_uint4((uint32_t)base, (uint32_t)nx | ((uint32_t)ny << 16) | (back ? kBackwards : 0u), t0, item);
    const bool neg = side ? (me.x & 0x80000000u) != 0 : (me.x & 0x8000u) != 0;
    s.side.x = __uint_as_float(side ? me.w : me.z);
    s.side.dx = neg ? -(float)g.F : (float)g.F;
    s.t_lo = __uint_as_float(t0);
    s.side.t_hi = __uint_as_float(me.y);
    const float2* cp = g.tpos + g.curve_pos[c];
    const uint32_t np = curve_slots(s.type);
    float p[4];
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
        float2 v = k < np ? cp[k] : make_float2(0.0f, 0.0f);
        p[k] = side ? v.y : v.x;
    }
    AxisPoly& a = s.side.a;
    a.p0 = p[0]; a.p1 = p[1]; a.p2 = p[2]; a.p3 = p[3];
    a.d01 = __fsub_rn(p[1], p[0]);
    a.d12 = __fsub_rn(p[2], p[1]);
    a.d23 = __fsub_rn(p[3], p[2]);
    s.side.inv = s.type == 2u && a.d01 != 0.0f ? __fdiv_rn(1.0f, a.d01) : 0.0f;
    return s;
}

// Work of the chains by tickets, longest class first: a ticket is a warp's
// share of a class (chain_share).  Built by every warp.
template <bool kSolve> struct ChainTickets {
    uint32_t start0, start1, n0, n1, first0, first1;   // two classes a lane
    uint32_t total;
    int32_t seg_log;
    SR_DEV uint32_t tickets_of(uint32_t n, uint32_t key) const {
        const ChainShare s = chain_share<kSolve>(key, seg_log);
        return s.lanes == 5 ? n << s.warps : ((n << s.lanes) + 31u) / 32u;
    }
    SR_DEV ChainShare share(uint32_t key) const { return chain_share<kSolve>(key, seg_log); }
    SR_DEV void build(const uint32_t* __restrict__ class_count, uint32_t sms) {
        const uint32_t lane = lane_id();
        seg_log = kSegLog;
        class_starts(class_count, start0, start1);
        n0 = class_count[2 * lane];
        n1 = class_count[2 * lane + 1];
        if (2 * lane + 1 == kEmptyPiece && kSolve) n1 = 0;
        if (kSolve) {
            const uint32_t t = __reduce_add_sync(0xFFFFFFFFu, tickets_of(n0, 2 * lane) + tickets_of(n1, 2 * lane + 1));
            seg_log = t < kShortTickets * sms ? kSegShort : (t >= kLongTickets * sms ? kSegLong : kSegLog);
        }
        const uint32_t t0 = tickets_of(n0, 2 * lane), t1 = tickets_of(n1, 2 * lane + 1);
        uint32_t x = t0 + t1;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, d);
            if ((int)lane >= d) x += y;
        }
        total = __shfl_sync(0xFFFFFFFFu, x, 31);
        first0 = x - t0 - t1;
        first1 = first0 + t0;
    }
    // The class of a ticket, this lane's chain of it (its list position; that
    // of the class's first chain, and false, for a lane without one) and which
    // of the chain's warps this is.
    SR_DEV bool find(uint32_t ticket, uint32_t list_cap, uint32_t& key, uint32_t& pos, uint32_t& warp) const {
        // the last class that starts at or before it (an empty class starts
        // where the next one does)
        const uint32_t m0 = __ballot_sync(0xFFFFFFFFu, first0 <= ticket);
        const uint32_t m1 = __ballot_sync(0xFFFFFFFFu, first1 <= ticket);
        const uint32_t at = 31u - (uint32_t)__clz((int)m0);
        const bool odd = (m1 >> at) & 1u;
        key = 2 * at + (odd ? 1u : 0u);
        const uint32_t tfirst = __shfl_sync(0xFFFFFFFFu, odd ? first1 : first0, at);
        const uint32_t cfirst = __shfl_sync(0xFFFFFFFFu, odd ? start1 : start0, at);
        const uint32_t ccount = __shfl_sync(0xFFFFFFFFu, odd ? n1 : n0, at);
        const ChainShare s = share(key);
        const uint32_t i = s.lanes == 5 ? (ticket - tfirst) >> s.warps : ((ticket - tfirst) * 32u + lane_id()) >> s.lanes;
        warp = (ticket - tfirst) & ((1u << s.warps) - 1u);
        const bool listed = i < ccount && cfirst + i < list_cap;
        pos = cfirst + (listed ? i : 0u);
        return listed;
    }
};

// A warp's first ticket, the CTAs being placed an SM after the other, `ctas`
// an SM: the first tickets go to as many SMs, the next ones to other
// schedulers of these (a CTA's warps are on different ones).  Tickets handed
// out by a counter from the start went to the SMs whose requests came first:
// of the 1,001 tickets of a 1024^2 frame six shared a scheduler and 3,000
// cycles a root, while others had none.
SR_DEV uint32_t first_ticket(uint32_t ctas) {
    const uint32_t sms = gridDim.x / ctas;
    return (blockIdx.x / sms * (blockDim.x / 32u) + (threadIdx.x >> 5)) * sms + blockIdx.x % sms;
}

__global__ void __launch_bounds__(128) k_chains(const GeomArgs g, const int32_t* __restrict__ offs,
                                                const uint4* __restrict__ pieces,
                                                const uint32_t* __restrict__ items, uint32_t list_cap,
                                                const uint32_t* __restrict__ class_count,
                                                uint32_t* __restrict__ queue, int32_t* __restrict__ cbuf,
                                                uint4* __restrict__ chain_piece) {
    wait_for_stream();
    ChainTickets<true> T;
    T.build(class_count, gridDim.x / kChainCtas);
    const uint32_t warps = gridDim.x * (blockDim.x / 32u);
    for (uint32_t ticket = first_ticket(kChainCtas); ticket < T.total;) {
        uint32_t key, pos, warp;
        const bool listed = T.find(ticket, list_cap, key, pos, warp);
        const ChainSetup s = chain_setup(g, offs, pieces, items[pos]);
        // a lane without a chain, or whose chain overflows (k_order_records
        // reports it), has no roots; a base below 0 is an offset past 2^31
        const int32_t len = listed && s.base >= 0 && s.base + s.len <= g.rec_cap ? s.len : 0;
        int32_t* out = cbuf + s.base;
        const uint32_t gl = T.share(key).lanes, cls = key & 3u;
        const int32_t lanes = 1 << gl, l = (int32_t)(lane_id() & ((1u << gl) - 1u));
        if (listed && l == 0) chain_piece[pos] = s.piece;
        if (cls == 0u) run_segments<4>(s.side, len, s.t_lo, out, lanes, l);
        else if (cls == 1u) run_segments<3>(s.side, len, s.t_lo, out, lanes, l);
        else if (cls == 2u) run_segments<2>(s.side, len, s.t_lo, out, lanes, l);
        else run_segments<(int)kArc>(s.side, len, s.t_lo, out, lanes, l);
        if (lane_id() == 0) ticket = warps + atomicAdd(queue, 1u);
        ticket = __shfl_sync(0xFFFFFFFFu, ticket, 0);
    }
}

// ------------------------------------------------------------- order -----
// The record order of make_intersection_1.comp:310-441: per piece, the
// start t0 and the two chains merged by `next_tx <= next_ty`, an exhausted
// side counting as 2.0 (with its side bit).  Roots never decrease along a
// chain (each is solved from the one before; only t0's flag bits may put it
// above the first ones), so a piece's records are the i0 x roots <= t0, then
// t0, then the stable merge (x first on ties) of the other x roots with the
// y roots, and a root's place is its index plus its rank in the other chain.
// A piece may run backwards: the fourth cut of a curve may lie before the
// third (make_intersection_0.comp:340).  Its roots never increase and stay
// below t0, and the sequential merge, which takes the lower head, takes all x
// roots, then t0, then all y roots: i0 is all of them.
//
// A lane finds the place of a root by a binary search; a warp's roots are
// neighbours, so its loads and stores are too.  The dependent loads bound it,
// of a chain's piece first: k_chains leaves it in one 16-byte word a chain (the
// curve's offset and its pieces summed up again took 0.184 instead of 0.158 ms
// on the 4096^2 frame of 21 M records, 0.127 instead of 0.106 in a batch of 64
// uneven scenes); then of the search, but a search by windows of 32 roots held
// by a warp, with a third of the loads, was no faster (0.197).  A thread per
// short and a CTA per long piece took 0.295; a lane walking a stretch of 16
// consecutive roots 0.52, its 4-byte accesses being scattered.
SR_DEV int32_t count_le(const int32_t* a, int32_t lo, int32_t hi, float v) {   // elements <= v, of a[lo, hi) sorted, + lo
    while (lo < hi) {
        const int32_t mid = (lo + hi) >> 1;
        if (bitsf(a[mid]) <= v) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}
SR_DEV int32_t count_lt(const int32_t* a, int32_t lo, int32_t hi, float v) {   // elements < v, likewise
    while (lo < hi) {
        const int32_t mid = (lo + hi) >> 1;
        if (bitsf(a[mid]) < v) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

__global__ void __launch_bounds__(128) k_order_records(const GeomArgs g, const int32_t* __restrict__ offs,
                                                       const uint4* __restrict__ pieces,
                                                       const uint32_t* __restrict__ items, uint32_t list_cap,
                                                       const uint32_t* __restrict__ class_count,
                                                       const uint4* __restrict__ chain_piece,
                                                       const int32_t* __restrict__ cbuf, int2* __restrict__ rec,
                                                       uint32_t* __restrict__ status) {
    wait_for_stream();
    ChainTickets<false> T;
    T.build(class_count, 0);
    const uint32_t warps = gridDim.x * (blockDim.x / 32u);
    for (uint32_t ticket = blockIdx.x * (blockDim.x / 32u) + (threadIdx.x >> 5); ticket < T.total; ticket += warps) {
        uint32_t key, pos, warp;
        if (!T.find(ticket, list_cap, key, pos, warp)) continue;
        // (k_chains left out the pieces without crossings)
        const uint4 pc = key == kEmptyPiece ? chain_setup(g, offs, pieces, items[pos]).piece : chain_piece[pos];
        const uint32_t item = pc.w, c = item >> 4;
        const int64_t base = (int64_t)pc.x;
        const int32_t nx = piece_nx(pc.y), ny = piece_ny(pc.y);
        if (base + 1 + nx + ny > g.rec_cap) {
            set_error(status, ERR_CAPACITY);
            continue;
        }
        const int32_t t0 = (int32_t)pc.z;
        const int32_t *X = cbuf + base + 1, *Y = X + nx;
        int2* R = rec + base;
        int32_t i0 = 0;
        const bool back = (pc.y & kBackwards) != 0;
        if (nx > 0 && ny > 0) {
            if (back) i0 = nx;
            else if (bitsf(X[0]) <= bitsf(t0)) i0 = count_le(X, 0, nx, bitsf(t0));
        }
        const uint32_t gl = T.share(key).lanes;
        const int32_t l = (int32_t)(lane_id() & ((1u << gl) - 1u));
        const bool y_side = (item & 1u) != 0;
        if (l == 0 && warp == 0 && (y_side || ny == 0)) R[i0] = make_int2((int32_t)c, t0);
        const int32_t len = y_side ? ny : nx, m = y_side ? nx : ny;
        const int32_t *A = y_side ? Y : X, *B = y_side ? X : Y;
        const int32_t k0 = (int32_t)warp * 256, k1 = imin(k0 + 256, len);
        int32_t r = 0;   // roots of the other chain before this one (x roots equal to a y root come before it)
        for (int32_t k = k0 + l; k < k1; k += 32) {
            const int32_t t = A[k];
            int32_t o;
            if (m == 0 || back) {
                o = k + (m == 0 ? 1 : (y_side ? 1 + nx : 0));
            } else if (y_side) {
                r = count_le(B, r, m, bitsf(t));
                o = 1 + k + imax(r, i0);
            } else {
                r = count_lt(B, r, m, bitsf(t));
                o = k < i0 ? k : 1 + k + r;
            }
            R[o] = make_int2((int32_t)c, stored_t(t));
        }
    }
}

// The reference's records for a read-back: the same order, found by the
// sequential merge itself, and the flags: a record whose t (flag bits masked)
// equals the previous one ORs the flags into both
// (make_intersection_1.comp:361-375).  A frame does not need them.
// Piece j of curve c, a thread each (pieces are merged independently: each
// starts from its own t0 and flag state).  The piece-0 thread also checks
// that the pieces cover the curve's records exactly.
SR_DEV void merge_piece(const GeomArgs& g, const int32_t* __restrict__ offs, const uint4* __restrict__ pieces,
                        const int32_t* __restrict__ cbuf, int2* __restrict__ rec, uint32_t* __restrict__ status,
                        uint32_t c, int j) {
    const int64_t start = offs[c], end = offs[c + 1];
    if (start >= end) return;
    if (start < 0 || end > g.rec_cap) {
        if (j == 0) set_error(status, ERR_CAPACITY);
        return;
    }
    const uint4* pt = pieces + (size_t)c * kMaxPieces;
    if (j == 0) {
        int64_t tot = start;
        for (int i = 0; i < kMaxPieces && tot < end; ++i) tot += 1 + piece_nx(pt[i].x) + piece_ny(pt[i].x);
        if (tot != end) set_error(status, ERR_RECORD_RANGE);
    }
    int64_t pc = start;
    for (int i = 0; i < j; ++i) pc += 1 + piece_nx(pt[i].x) + piece_ny(pt[i].x);
    if (pc >= end) return;   // the curve has fewer pieces
    const uint4 me = pt[j];
    const int32_t nx = piece_nx(me.x), ny = piece_ny(me.x);
    const int32_t n_loop = nx + ny + 1;
    if (pc + n_loop > end) return;   // reported by the piece-0 thread
    const int32_t t0 = j == 0 ? 0 : (int32_t)pt[j - 1].y;   // bits of 0.0f for the first piece
    const int32_t minus_one = fbits(-1.0f);
    const int32_t ex_x = fbits(2.0f), ex_y = fbits(2.0f) | 1;
    const int32_t* X = cbuf + pc + 1;
    const int32_t* Y = X + nx;
    // heads: A = x side, B = y side (make_intersection_1.comp:321-359)
    int32_t ia = 0, ib = 0;
    // both sides cross: A = x chain, B = [t0, y chain]; no x crossing:
    // A empty, B = [t0, y chain]; no y crossing: A = [t0, x chain], B empty
    const bool a_has_t0 = (nx > 0 && ny == 0);
    const int32_t lenA = nx + (a_has_t0 ? 1 : 0);
    const int32_t lenB = a_has_t0 ? 0 : ny + 1;
    int32_t last = minus_one;
    for (int32_t k = 0; k < n_loop; ++k) {
        int32_t av = ex_x, bv = ex_y;
        if (ia < lenA) av = a_has_t0 ? (ia == 0 ? t0 : X[ia - 1]) : X[ia];
        if (ib < lenB) bv = ib == 0 ? t0 : Y[ib - 1];
        int32_t out;
        if (bitsf(av) <= bitsf(bv)) {
            out = av;
            ++ia;
        } else {
            out = stored_t(bv);
            ++ib;
        }
        if ((out & ~3) == (last & ~3)) {
            out |= last;
            rec[pc - 1] = make_int2((int32_t)c, out);
        }
        rec[pc] = make_int2((int32_t)c, out);
        last = out;
        ++pc;
    }
}

// A thread per (curve, piece).
__global__ void __launch_bounds__(128) k_merge(const GeomArgs g, const int32_t* __restrict__ offs,
                                               const uint4* __restrict__ pieces, const int32_t* __restrict__ cbuf,
                                               int2* __restrict__ rec, uint32_t* __restrict__ status) {
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t c = tid / kMaxPieces;
    if (c < g.n_curves) merge_piece(g, offs, pieces, cbuf, rec, status, c, (int)(tid % kMaxPieces));
}

// ---------------------------------------------------------- fragment -----
// gen_fragment.comp:90-245, a lane per record: the piece between this
// record's t and the next record's t (t = 1 when the next record belongs to
// another curve), its cell, the 64-bit sort key, the winding change across
// the sample row and (pixel mode) the part of it left of the cell centre.
// A warp takes 32 consecutive records and writes the first 31: each lane
// evaluates the curve at its own record, and the next lane's point (or the
// curve's end, from the count pass) is the piece's end.  Instruction issue
// and the latency of the curve's loads bound it: 0.206 ms on the 4096^2 frame
// of 21 M records, 0.122 in a batch of 64 uneven scenes (CTAs of eight warps
// 0.208 and 0.128; evaluating both ends in every lane took 0.225).
constexpr int kFragWarps = 4, kFragOut = 31;

// SEG: the first seg_ctas CTAs build the tables of the per-path sort beside
// that.  For a frame of few paths that saves the tables' launch, 3 us of the 154
// of the 1024^2 frame; of many paths the kernel with the call in it is slower by
// as much as the launch takes (0.212 instead of 0.205 ms on the 4096^2 frame).
constexpr uint32_t kSegPaths = 4096;
static_assert(kSegThreads == 32 * kFragWarps, "one launch");
template <bool SEG>
__global__ void __launch_bounds__(32 * kFragWarps) k_fragment(
    const GeomArgs g, const int2* __restrict__ rec, int64_t n_cap, const uint32_t* __restrict__ n_dev,
    uint64_t* __restrict__ keys, uint8_t* __restrict__ wnp, DebugOut dbg, uint32_t seg_ctas,
    const __grid_constant__ SegArgs seg, const __grid_constant__ TileTables tables, uint32_t* status, uint32_t spin_limit) {
    wait_for_stream();
    if (SEG && blockIdx.x < seg_ctas) {
        seg_tiles(seg, tables, status, spin_limit);
        return;
    }
    const int64_t n = (int64_t)min((uint64_t)*n_dev, (uint64_t)n_cap);
    const int64_t b = ((int64_t)(blockIdx.x - (SEG ? seg_ctas : 0u)) * kFragWarps + (threadIdx.x >> 5)) * kFragOut;
    if (b >= n) return;
    const uint32_t lane = lane_id();
    const int64_t i = b + lane;
    const int2 r = i < n ? rec[i] : make_int2(-1, 0);
    const uint32_t c = (uint32_t)r.x;
    // an index out of range only in a frame whose records overflowed their
    // capacity (it is reported and discarded)
    const bool ok = c < g.n_curves;
    const float t0 = gmax(bitsf(r.y & ~3), 0.0f);
    uint32_t path = 0;
    float2 pf = make_float2(0.0f, 0.0f);
    if (ok) {
        const uint32_t type = g.curve_type[c];
        path = g.curve_path[c];
        CurvePts P;
        load_curve(g.tpos, g.curve_pos[c], type, P);
        pf = make_float2(curve_coord(type, t0, P.x), curve_coord(type, t0, P.y));
    }
    const bool more = __shfl_down_sync(0xFFFFFFFFu, c, 1) == c;
    float t1 = __shfl_down_sync(0xFFFFFFFFu, t0, 1);
    float2 pl = make_float2(__shfl_down_sync(0xFFFFFFFFu, pf.x, 1), __shfl_down_sync(0xFFFFFFFFu, pf.y, 1));
    if (lane == 31 || i >= n) return;
    if (!ok) {
        keys[i] = ~0ull;
        if (wnp) wnp[i] = 0;
        return;
    }
    if (!more) {
        t1 = 1.0f;
        pl = g.curve_end[c];
    }
    int32_t yx = (int32_t)0xFFFEFFFE, wn = 0, left = 0;
    bool valid = false;
    int32_t pos_x = 0, pos_y = 0;
    if (t0 < t1) {
        const int32_t F = g.F;
        int32_t W = g.W, H = g.H;
        if (g.st.n_scenes > 1) {
            const SceneInfo& si = scene_of_path(g.st, path);
            W = si.W;
            H = si.H;
        }
        const float invF = inv_F(F);
        int32_t rx = wmul(float2int_rd(__fmul_rn(__fmul_rn(__fadd_rn(pf.x, pl.x), 0.5f), invF)), F);
        int32_t ry = wmul(float2int_rd(__fmul_rn(__fmul_rn(__fadd_rn(pf.y, pl.y), 0.5f), invF)), F);
        pos_x = imin(imax(rx, -F), wadd(W & (int32_t)0xFFFFFFFE, F));
        pos_y = imin(imax(ry, -F), wadd(H & (int32_t)0xFFFFFFFE, F));
        if ((uint32_t)ry < (uint32_t)H) {
            valid = true;
            yx = (int32_t)(((uint32_t)wadd(pos_y, 0x7FFF) << 16) | ((uint32_t)wadd(pos_x, 0x7FFF) & 0xFFFFu));
        }
        // winding sample row cell_y + FRAG_SIZE/2 (gen_fragment.comp:188-199)
        float wn_y = __fadd_rn((float)pos_y, __fmul_rn(0.5f, (float)F));
        if (pf.y == pl.y) wn = 0;
        else if (pf.y < wn_y && wn_y <= pl.y) wn = -1;
        else if (pl.y < wn_y && wn_y <= pf.y) wn = 1;
        if (g.pixel_mode && wn != 0) {
            float dyv = __fsub_rn(pl.y, pf.y);
            float tc = __fdiv_rn(__fsub_rn(wn_y, pf.y), dyv);
            float xc = __fadd_rn(pf.x, __fmul_rn(tc, __fsub_rn(pl.x, pf.x)));
            if (xc < __fadd_rn((float)pos_x, 0.5f)) left = wn;
        }
    }
    const uint32_t wbits = (uint32_t)((wn & 3) | ((left & 3) << 2));
    const uint64_t key = pack_key(g.L, path, valid, pos_y, pos_x);
    if (wnp) {
        keys[i] = key;
        wnp[i] = (uint8_t)wbits;
    } else {
        keys[i] = key | ((uint64_t)wbits << key_bits(g.L));   // winding bits ride above the key
    }
    if (dbg.fkey) {
        dbg.fkey[i] = yx;
        dbg.fwn[i] = wn;
        dbg.fleft[i] = left;
    }
}

// -------------------------------------------------------------- launches --
void launch_arc_fixup(const uint32_t* curve_type, const uint32_t* curve_pos, const uint32_t* curve_path,
                      uint32_t n_curves, const float2* pos, const SceneTable& t, float2* tpos, int32_t* path_visible,
                      cudaStream_t st) {
    if (n_curves == 0) return;
    count_launches(1);
    launch_after(k_arc_fixup, (n_curves + 255) / 256, 256, 0, st, curve_type, curve_pos, curve_path, n_curves, pos, t,
                 tpos, path_visible);
}

void launch_transform(const float2* pos, const uint32_t* pos_path, uint32_t n_points, const SceneTable& t,
                      float2* tpos, int32_t* path_visible, void* zero, size_t zero_bytes, int sm_count,
                      cudaStream_t st) {
    const size_t words = zero_bytes / 16, clear = std::min<size_t>((words + 1023) / 1024, (size_t)std::max(sm_count, 1) * 4);
    const unsigned grid = std::max((n_points + 255) / 256, (uint32_t)clear);
    if (grid == 0) return;
    count_launches(1);
    launch_after(k_transform, grid, 256, 0, st, pos, pos_path, n_points, t, tpos, path_visible,
                 static_cast<uint4*>(zero), words);
}

size_t piece_table_bytes(uint32_t n_curves) { return sizeof(uint4) * kMaxPieces * (size_t)n_curves; }
uint32_t chain_list_capacity(uint32_t n_curves) { return 2u * kMaxPieces * n_curves; }

void launch_count(const GeomArgs& g, float* cut_cache, int32_t* count, const ChainWork& w, uint32_t* status,
                  cudaStream_t st) {
    if (g.n_curves == 0) return;
    count_launches(1);
    if (g.n_curves <= kFewCurves)
        launch_after(k_count<8>, (8 * g.n_curves + kCountThreads - 1) / kCountThreads, kCountThreads, 0, st, g,
                     cut_cache, count, w.pieces, w.chain_items, w.chain_keys, w.list_cap, w.chain_count, w.class_count,
                     status);
    else
        launch_after(k_count<1>, (g.n_curves + kCountThreads - 1) / kCountThreads, kCountThreads, 0, st, g, cut_cache,
                     count, w.pieces, w.chain_items, w.chain_keys, w.list_cap, w.chain_count, w.class_count, status);
}

static uint32_t offset_tiles(uint32_t n_curves) { return (n_curves + 1024 * kOffsetRows - 1) / (1024 * kOffsetRows); }
size_t offset_scan_words(uint32_t n_curves) { return (size_t)offset_tiles(n_curves) + 1; }

void launch_offsets_and_order(const GeomArgs& g, const int32_t* count, int32_t* offs, const ChainWork& w,
                              uint64_t* tile_status, uint32_t* tile_counter, uint32_t* report_n, uint32_t* status,
                              int sm_count, cudaStream_t st) {
    if (g.n_curves == 0) {
        cudaMemsetAsync(offs, 0, sizeof(int32_t), st);
        return;
    }
    count_launches(1);
    const uint32_t tiles = offset_tiles(g.n_curves);
    const unsigned order = (unsigned)std::min<size_t>(((size_t)w.list_cap + 255) / 256, (size_t)sm_count * 4);
    launch_after(k_offsets_and_order, tiles + order, 256, 0, st, count, offs, g.n_curves, tiles, tile_status,
                 tile_counter, report_n, status, spin_limit(), w.chain_items, w.chain_keys, w.list_cap, w.chain_count,
                 w.class_count, w.class_next, w.sorted_items);
}

void launch_chains(const GeomArgs& g, const int32_t* offs, const ChainWork& w, int32_t* cbuf, int sm_count,
                   cudaStream_t st) {
    if (g.n_curves == 0) return;
    count_launches(1);
    // (not launch_after: placed while the offset scan drains, its CTAs do not
    // spread over the SMs, 1,725 instead of 1,675 us for a 4096^2 frame)
    k_chains<<<sm_count * kChainCtas, 128, 0, st>>>(g, offs, w.pieces, w.sorted_items, w.list_cap, w.class_count,
                                                    w.chain_queue, cbuf, w.chain_piece);
}

void launch_merge(const GeomArgs& g, const int32_t* offs, const ChainWork& w, const int32_t* cbuf, int2* rec,
                  uint32_t* status, cudaStream_t st) {
    if (g.n_curves == 0) return;
    count_launches(1);
    k_merge<<<(unsigned)(((size_t)g.n_curves * kMaxPieces + 127) / 128), 128, 0, st>>>(g, offs, w.pieces, cbuf, rec,
                                                                                       status);
}

void launch_order_records(const GeomArgs& g, const int32_t* offs, const ChainWork& w, const int32_t* cbuf, int2* rec,
                          uint32_t* status, int sm_count, cudaStream_t st) {
    if (g.n_curves == 0) return;
    count_launches(1);
    launch_after(k_order_records, sm_count * 32, 128, 0, st, g, offs, w.pieces, w.sorted_items, w.list_cap,
                 w.class_count, w.chain_piece, cbuf, rec, status);
}

void launch_fragment(const GeomArgs& g, const int2* rec, int64_t n_cap, const uint32_t* n_dev, uint64_t* keys,
                     uint8_t* wnp, DebugOut dbg, SegArgs* seg, uint32_t* status, cudaStream_t st) {
    if (n_cap <= 0 || g.n_curves == 0) return;
    count_launches(1);
    constexpr int64_t per = kFragWarps * kFragOut;
    const unsigned grid = (unsigned)((n_cap + per - 1) / per);
    if (seg && seg->n_paths <= kSegPaths) {
        const uint32_t seg_ctas = (seg->n_paths + kSegThreads - 1) / kSegThreads;
        seg->tables_built = true;
        launch_after(k_fragment<true>, grid + seg_ctas, 32 * kFragWarps, 0, st, g, rec, n_cap, n_dev, keys, wnp, dbg,
                     seg_ctas, *seg, segsort_tables(*seg), status, spin_limit());
    } else {
        launch_after(k_fragment<false>, grid, 32 * kFragWarps, 0, st, g, rec, n_cap, n_dev, keys, wnp, dbg, 0u,
                     SegArgs{}, TileTables{}, status, spin_limit());
    }
}

}  // namespace sr
