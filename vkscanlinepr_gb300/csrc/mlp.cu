// mlp.cu — learned buffer sizing: path features, labels, and a small MLP
// trained and run by hand-written kernels.
//
// The reference sizes its intersection and fragment buffers by reading the
// count pass back to the host every frame (scanline_rasterizer.cpp:337-369,
// :578-584).  Here a 6-64-64-2 GELU network predicts, per path, log(1 + the
// number of intersection records) and log(1 + the number of draw records)
// from cheap features of its control points, so a frame can be sized when
// its scenes are uploaded and then enqueued without that read-back.  The
// prediction changes allocation only; an overflow is detected on the device
// and the frame reruns with exact sizing.
//
// Weights are BF16 (an FP32 master copy is kept for Adam); every product is
// accumulated in FP32.  Layout of the packed parameter vector:
//   W1[64][6] b1[64] W2[64][64] b2[64] W3[2][64] b3[2]
// Inputs and targets are standardised with a fixed normaliser
//   norm = x_mean[6] x_inv_std[6] y_mean[2] y_std[2]
// so the network works in standard units; predictions are returned in
// log(1 + count) units.
#include <atomic>

#include <cuda_bf16.h>

#include "common.cuh"
#include "kernels.h"

namespace sr {

namespace {
constexpr int kIn = kMlpIn, kH = kMlpHidden, kOut = kMlpOut;
constexpr int oW1 = 0, oB1 = oW1 + kH * kIn, oW2 = oB1 + kH, oB2 = oW2 + kH * kH, oW3 = oB2 + kH,
              oB3 = oW3 + kOut * kH, kParams = oB3 + kOut;
static_assert(kParams == kMlpParams, "parameter layout");
constexpr int nXm = 0, nXs = kIn, nYm = 2 * kIn, nYs = 2 * kIn + kOut;
static_assert(nYs + kOut == kMlpNorm, "normaliser layout");
// Shared-memory copies of the parameters: weights rounded to BF16 as the
// forward pass uses them, biases FP32.  W1 is transposed (neighbouring lanes
// take neighbouring units); a row of W2, as of the activations, is padded to
// 68 floats, so that 16-byte reads of eight neighbouring rows meet no bank
// twice.
constexpr int kRow = kH + 4;
struct Params {
    __align__(16) float w2[kH][kRow];
    __align__(16) float w1t[kIn][kH];
    __align__(16) float w3[kOut][kH];
    __align__(16) float b1[kH], b2[kH];
    float b3[kOut];
    float norm[kMlpNorm];
};

SR_DEV float gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }
// d/dx [x Phi(x)] = Phi(x) + x phi(x)
SR_DEV float gelu_grad(float x) {
    const float cdf = 0.5f * (1.0f + erff(x * 0.70710678118654752f));
    const float pdf = 0.39894228040143268f * expf(-0.5f * x * x);
    return fmaf(x, pdf, cdf);
}

SR_DEV float bf(const __nv_bfloat16& w) { return __bfloat162float(w); }
SR_DEV void load_params(const __nv_bfloat16* __restrict__ wb, const float* __restrict__ master,
                        const float* __restrict__ norm, Params& P) {
    const int tid = threadIdx.x, nt = blockDim.x;
    static_assert(oW2 % 8 == 0 && kH % 8 == 0, "16-byte reads of W2");
    for (int i = tid; i < kH * kH / 8; i += nt) {
        const uint4 v = reinterpret_cast<const uint4*>(wb + oW2)[i];
        const uint32_t u[4] = {v.x, v.y, v.z, v.w};
        float4 f[2];
        float* q = reinterpret_cast<float*>(f);
#pragma unroll
        for (int k = 0; k < 4; ++k) {   // a BF16 is the upper half of its float
            q[2 * k] = __uint_as_float(u[k] << 16);
            q[2 * k + 1] = __uint_as_float(u[k] & 0xFFFF0000u);
        }
        float4* row = reinterpret_cast<float4*>(&P.w2[8 * i / kH][8 * i % kH]);
        row[0] = f[0];
        row[1] = f[1];
    }
    for (int i = tid; i < kH * kIn; i += nt) P.w1t[i % kIn][i / kIn] = bf(wb[oW1 + i]);
    for (int i = tid; i < kOut * kH; i += nt) P.w3[i / kH][i % kH] = bf(wb[oW3 + i]);
    for (int i = tid; i < kH; i += nt) {
        P.b1[i] = master[oB1 + i];
        P.b2[i] = master[oB2 + i];
    }
    if (tid < kOut) P.b3[tid] = master[oB3 + tid];
    if (tid < kMlpNorm) P.norm[tid] = norm[tid];
}
}  // namespace

// ------------------------------------------------------------ features ---
// Per path, from its transformed control points: segment count, bounding
// box clipped to one pixel around its canvas, control-polygon length, sum of
// absolute turning angles between successive control-polygon edges, and the
// fraction of cubic segments.  Lengths are in cells; counts, lengths and the
// turn sum enter as log(1 + x).
__global__ void k_path_features(const GeomArgs g, const uint32_t* __restrict__ path_first_curve, uint32_t n_paths,
                                float* __restrict__ feats) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n_paths) return;
    const SceneInfo& si = scene_of_path(g.st, p);
    const float W = (float)si.W, H = (float)si.H;
    const uint32_t c0 = path_first_curve[p], c1 = path_first_curve[p + 1];
    float xmin = 3.0e38f, ymin = 3.0e38f, xmax = -3.0e38f, ymax = -3.0e38f;
    float len = 0.0f, turn = 0.0f;
    uint32_t cubics = 0;
    float pex = 0.0f, pey = 0.0f;   // previous non-degenerate edge
    bool have_edge = false;
    for (uint32_t c = c0; c < c1; ++c) {
        const uint32_t type = g.curve_type[c];
        const uint32_t np = type & 7u;
        const float2* cp = g.tpos + g.curve_pos[c];
        cubics += type == 4u ? 1u : 0u;
        float2 a = cp[0];
        xmin = fminf(xmin, a.x); xmax = fmaxf(xmax, a.x);
        ymin = fminf(ymin, a.y); ymax = fmaxf(ymax, a.y);
        for (uint32_t k = 1; k < np; ++k) {
            const float2 b = cp[k];
            xmin = fminf(xmin, b.x); xmax = fmaxf(xmax, b.x);
            ymin = fminf(ymin, b.y); ymax = fmaxf(ymax, b.y);
            const float ex = b.x - a.x, ey = b.y - a.y;
            const float el = sqrtf(ex * ex + ey * ey);
            if (el > 0.0f) {
                len += el;
                if (have_edge) turn += fabsf(atan2f(pex * ey - pey * ex, pex * ex + pey * ey));
                pex = ex;
                pey = ey;
                have_edge = true;
            }
            a = b;
        }
    }
    const uint32_t segs = c1 - c0;
    float bw = 0.0f, bh = 0.0f;
    if (segs) {
        bw = fmaxf(fminf(xmax, W + 1.0f) - fmaxf(xmin, -1.0f), 0.0f);
        bh = fmaxf(fminf(ymax, H + 1.0f) - fmaxf(ymin, -1.0f), 0.0f);
    }
    const float invF = inv_F(g.F);
    float* f = feats + (size_t)p * kIn;
    f[0] = log1pf((float)segs);
    f[1] = log1pf(bw * invF);
    f[2] = log1pf(bh * invF);
    f[3] = log1pf(fminf(len, 1.0e30f) * invF);
    f[4] = log1pf(turn * 0.15915494309189535f);   // in turns
    f[5] = segs ? (float)cubics / (float)segs : 0.0f;
}

// Per path: log(1 + records) from the count pass and log(1 + draw records)
// from the emit's per-path counters.
__global__ void k_path_labels(const uint32_t* __restrict__ path_first_curve, uint32_t n_paths,
                              const int32_t* __restrict__ count, const uint32_t* __restrict__ path_draw,
                              float* __restrict__ labels) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n_paths) return;
    int64_t n = 0;
    for (uint32_t c = path_first_curve[p]; c < path_first_curve[p + 1]; ++c) n += count[c];
    labels[(size_t)p * kOut + 0] = log1pf((float)n);
    labels[(size_t)p * kOut + 1] = log1pf((float)path_draw[p]);
}

// ------------------------------------------------------------ inference --
// A warp takes eight paths, a lane two of the 64 units of each layer for all
// eight: a weight read from shared memory serves eight multiply-adds, and 16
// sums are in flight a lane.  The second layer's multiply-adds are done two
// paths an instruction (fma.rn.f32x2, each half rounded as fmaf).  Instruction
// issue bounds it (128 erf a path are the larger part): 200,000 paths take 62.6
// us, 20,000 take 12.0 and 5,000 take 6.5; with an instruction a multiply-add
// 67.3 for 200,000, with four CTAs an SM and 64 registers 61.6, but 14.5 for
// 20,000; with sixteen paths a warp 64.4; a path a thread (64 values in 247
// registers, one sum in flight) took 141, and 27 for 5,000.
// Two floats in one register pair, and a * b + c of both (rounded as fmaf).
SR_DEV uint64_t pair(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
SR_DEV void unpair(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
SR_DEV uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

constexpr int kPredictThreads = 256, kPredictCtas = 3, kWarpPaths = 8;
struct PredictSmem {
    Params P;
    __align__(16) float h[kPredictThreads / 32][kH][kWarpPaths];   // a unit's values of the warp's paths
};
__global__ void __launch_bounds__(kPredictThreads, kPredictCtas) k_mlp_predict(
    const __nv_bfloat16* __restrict__ wb, const float* __restrict__ master, const float* __restrict__ norm,
    const float* __restrict__ x, uint32_t n, float* __restrict__ y) {
    wait_for_stream();
    __shared__ PredictSmem S;
    const Params& P = S.P;
    load_params(wb, master, norm, S.P);
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float(*h)[kWarpPaths] = S.h[warp];
    const uint32_t warps = gridDim.x * (kPredictThreads / 32), groups = n / kWarpPaths + (n % kWarpPaths ? 1u : 0u);
    for (uint32_t g = blockIdx.x * (kPredictThreads / 32) + warp; g < groups; g += warps) {
        const int here = g < n / kWarpPaths ? kWarpPaths : (int)(n % kWarpPaths);   // paths of this group
        const float* xg = x + (size_t)g * (kWarpPaths * kIn);   // (6 n needs more than 32 bits)
        // layer 1: units lane and lane + 32
        float v0 = 0.0f, v1 = 0.0f;   // the eight paths' 48 inputs, standardised
        {
            const int k0 = lane % kIn, k1 = (lane + 32) % kIn;
            if (lane < here * kIn) v0 = (xg[lane] - P.norm[nXm + k0]) * P.norm[nXs + k0];
            if (lane + 32 < here * kIn) v1 = (xg[lane + 32] - P.norm[nXm + k1]) * P.norm[nXs + k1];
        }
#pragma unroll
        for (int q0 = 0; q0 < kWarpPaths; q0 += 4) {
            float4 g0, g1;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float a0 = P.b1[lane], a1 = P.b1[lane + 32];
#pragma unroll
                for (int k = 0; k < kIn; ++k) {
                    const int e = (q0 + i) * kIn + k;
                    const float in = __shfl_sync(0xFFFFFFFFu, e < 32 ? v0 : v1, e & 31);
                    a0 = fmaf(P.w1t[k][lane], in, a0);
                    a1 = fmaf(P.w1t[k][lane + 32], in, a1);
                }
                (&g0.x)[i] = gelu(a0);
                (&g1.x)[i] = gelu(a1);
            }
            *reinterpret_cast<float4*>(&h[lane][q0]) = g0;
            *reinterpret_cast<float4*>(&h[lane + 32][q0]) = g1;
        }
        __syncwarp();
        // layer 2, two paths an instruction
        uint64_t s0[kWarpPaths / 2], s1[kWarpPaths / 2];
#pragma unroll
        for (int q = 0; q < kWarpPaths / 2; ++q) {
            s0[q] = pair(P.b2[lane], P.b2[lane]);
            s1[q] = pair(P.b2[lane + 32], P.b2[lane + 32]);
        }
#pragma unroll 2
        for (int k = 0; k < kH; k += 4) {
            const float4 w0 = *reinterpret_cast<const float4*>(&P.w2[lane][k]);
            const float4 w1 = *reinterpret_cast<const float4*>(&P.w2[lane + 32][k]);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint64_t d0 = pair((&w0.x)[i], (&w0.x)[i]), d1 = pair((&w1.x)[i], (&w1.x)[i]);
#pragma unroll
                for (int q = 0; q < kWarpPaths / 2; q += 2) {
                    const ulonglong2 u = *reinterpret_cast<const ulonglong2*>(&h[k + i][2 * q]);
                    s0[q] = fma2(d0, u.x, s0[q]);
                    s1[q] = fma2(d1, u.x, s1[q]);
                    s0[q + 1] = fma2(d0, u.y, s0[q + 1]);
                    s1[q + 1] = fma2(d1, u.y, s1[q + 1]);
                }
            }
        }
        float a0[kWarpPaths], a1[kWarpPaths];
#pragma unroll
        for (int q = 0; q < kWarpPaths / 2; ++q) {
            unpair(s0[q], a0[2 * q], a0[2 * q + 1]);
            unpair(s1[q], a1[2 * q], a1[2 * q + 1]);
        }
        // layer 3: 16 sums over the lanes, halving the sums a lane holds with
        // every exchange: lane l ends with output l & 15 (path l / 2 & 7,
        // output l & 1), the two halves of the warp added last
        float o[2 * kWarpPaths];
        const float w30 = P.w3[0][lane], w31 = P.w3[0][lane + 32], w40 = P.w3[1][lane], w41 = P.w3[1][lane + 32];
#pragma unroll
        for (int q = 0; q < kWarpPaths; ++q) {
            const float g0 = gelu(a0[q]), g1 = gelu(a1[q]);
            o[2 * q] = fmaf(w31, g1, w30 * g0);
            o[2 * q + 1] = fmaf(w41, g1, w40 * g0);
        }
#pragma unroll
        for (int d = 8; d; d >>= 1) {
            const bool up = (lane & d) != 0;
#pragma unroll
            for (int i = 0; i < d; ++i) {
                const float mine = up ? o[i + d] : o[i], other = up ? o[i] : o[i + d];
                o[i] = mine + __shfl_xor_sync(0xFFFFFFFFu, other, d);
            }
        }
        const float sum = o[0] + __shfl_xor_sync(0xFFFFFFFFu, o[0], 16);
        const int k = lane & 1;
        if (lane < here * kOut)
            y[(size_t)g * (kWarpPaths * kOut) + lane] = fmaf(sum + P.b3[k], P.norm[nYs + k], P.norm[nYm + k]);
        __syncwarp();
    }
}

// ------------------------------------------------------------- training --
// Adam on the FP32 master copy (bias-corrected moments); refreshes the BF16
// weights and clears the gradient for the next step.
struct AdamArgs {
    float *master, *m, *v;
    __nv_bfloat16* wb;
    float lr, b1, b2, eps, bc1, bc2;
};
// By a CTA of kThreads; every load before the first store, so that they are
// in flight together.
template <int kThreads> SR_DEV void adam_all(const AdamArgs& A, float* grad) {
    constexpr int K = (kParams + kThreads - 1) / kThreads;
    float g[K], m[K], v[K], w[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int i = threadIdx.x + k * kThreads;
        if (i >= kParams) continue;
        g[k] = __ldcg(grad + i);
        m[k] = A.m[i];
        v[k] = A.v[i];
        w[k] = A.master[i];
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int i = threadIdx.x + k * kThreads;
        if (i >= kParams) continue;
        const float mi = A.b1 * m[k] + (1.0f - A.b1) * g[k];
        const float vi = A.b2 * v[k] + (1.0f - A.b2) * g[k] * g[k];
        A.m[i] = mi;
        A.v[i] = vi;
        const float wi = w[k] - A.lr * (mi / A.bc1) / (sqrtf(vi / A.bc2) + A.eps);
        A.master[i] = wi;
        A.wb[i] = __float2bfloat16_rn(wi);
        grad[i] = 0.0f;
    }
}

SR_DEV void red_add4(float* p, float a, float b, float c, float d) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

// Forward and backward of the mean squared error (in standard units) over
// one minibatch: rows idx[0..n) of (x, t), or rows 0..n when idx is NULL.
// A CTA takes 32 samples: a minibatch of 4,096 is 128 CTAs, one wave with 16
// warps on an SM.  Every layer is a small product out of shared memory in
// which a thread owns 2 to 8 outputs, read in 16-byte pieces; the CTA's
// parameter gradients are summed over its samples in registers and added into
// grad.  loss_sum receives the sum of squared errors (a double: a float sum
// in the order the warps come differs by up to 3e-6 from run to run).  With
// `adam`, the CTA that finishes last takes the optimiser step (a launch and its
// gap saved).
// Shared-memory reads and the latency of its eight phases bound it: 16 steps
// of 4,096 samples and the two shuffles before them take 515 us, where 64 CTAs
// of 64 threads, a sample each, and a separate optimiser launch took 1,740.
constexpr int kSamples = 32, kGradThreads = 512;
struct GradSmem {
    Params P;
    __align__(16) float a1[kSamples][kRow], h1[kSamples][kRow], a2[kSamples][kRow], h2[kSamples][kRow];
    __align__(16) float d2[kSamples][kRow], d1[kSamples][kRow];
    float xin[kSamples][kIn];
    float ty[kSamples][kOut];   // standardised targets
    float dy[kSamples][kOut];
    bool last;
};

// Row of sample i.  (A shuffle whose sort gave up, which the caller is told at
// the end, leaves places of the order unwritten: what they hold may be no row.)
SR_DEV uint32_t sample_row(const uint32_t* __restrict__ idx, uint32_t rows, uint32_t i) {
    return idx ? min(idx[i], rows - 1u) : i;
}

__global__ void __launch_bounds__(kGradThreads) k_mlp_grad(const __nv_bfloat16* __restrict__ wb,
                                                           const float* __restrict__ master,
                                                           const float* __restrict__ norm, const float* __restrict__ x,
                                                           const float* __restrict__ t,
                                                           const uint32_t* __restrict__ idx, uint32_t rows, uint32_t n,
                                                           float scale,
                                                           float* grad, double* loss_sum, int adam, AdamArgs A,
                                                           uint32_t* done) {
    wait_for_previous();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    GradSmem& S = *reinterpret_cast<GradSmem*>(smem_raw);
    const Params& P = S.P;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t s0 = blockIdx.x * kSamples;
    load_params(wb, master, norm, S.P);
    if (tid < kSamples * kIn) {
        const int q = tid / kIn, k = tid % kIn;
        const uint32_t sidx = s0 + q;
        float v = 0.0f;
        if (sidx < n) v = (x[(size_t)sample_row(idx, rows, sidx) * kIn + k] - norm[nXm + k]) * norm[nXs + k];
        S.xin[q][k] = v;
    } else if (tid >= kGradThreads - kSamples * kOut) {
        const int i = tid - (kGradThreads - kSamples * kOut), q = i / kOut, k = i % kOut;
        const uint32_t sidx = s0 + q;
        float v = 0.0f;
        if (sidx < n) v = (t[(size_t)sample_row(idx, rows, sidx) * kOut + k] - norm[nYm + k]) / norm[nYs + k];
        S.ty[q][k] = v;
    }
    __syncthreads();
    // layer 1: 4 outputs a thread
#pragma unroll
    for (int i = 0; i < kSamples * kH / kGradThreads; ++i) {
        const int q = (tid + i * kGradThreads) / kH, j = tid % kH;
        float a = P.b1[j];
#pragma unroll
        for (int k = 0; k < kIn; ++k) a = fmaf(P.w1t[k][j], S.xin[q][k], a);
        S.a1[q][j] = a;
        S.h1[q][j] = gelu(a);
    }
    __syncthreads();
    // layer 2: two units of two samples a thread
    {
        const int q = 2 * warp, j = lane;
        float a00 = P.b2[j], a01 = P.b2[j + 32], a10 = a00, a11 = a01;
#pragma unroll 4
        for (int k = 0; k < kH; k += 4) {
            const float4 u = *reinterpret_cast<const float4*>(&S.h1[q][k]);
            const float4 v = *reinterpret_cast<const float4*>(&S.h1[q + 1][k]);
            const float4 w0 = *reinterpret_cast<const float4*>(&P.w2[j][k]);
            const float4 w1 = *reinterpret_cast<const float4*>(&P.w2[j + 32][k]);
            a00 = fmaf(w0.x, u.x, a00); a01 = fmaf(w1.x, u.x, a01); a10 = fmaf(w0.x, v.x, a10); a11 = fmaf(w1.x, v.x, a11);
            a00 = fmaf(w0.y, u.y, a00); a01 = fmaf(w1.y, u.y, a01); a10 = fmaf(w0.y, v.y, a10); a11 = fmaf(w1.y, v.y, a11);
            a00 = fmaf(w0.z, u.z, a00); a01 = fmaf(w1.z, u.z, a01); a10 = fmaf(w0.z, v.z, a10); a11 = fmaf(w1.z, v.z, a11);
            a00 = fmaf(w0.w, u.w, a00); a01 = fmaf(w1.w, u.w, a01); a10 = fmaf(w0.w, v.w, a10); a11 = fmaf(w1.w, v.w, a11);
        }
        S.a2[q][j] = a00; S.a2[q][j + 32] = a01; S.a2[q + 1][j] = a10; S.a2[q + 1][j + 32] = a11;
        S.h2[q][j] = gelu(a00); S.h2[q][j + 32] = gelu(a01);
        S.h2[q + 1][j] = gelu(a10); S.h2[q + 1][j + 32] = gelu(a11);
    }
    __syncwarp();
    // layer 3 and the error: a warp its two samples, a lane two units of each
    {
        float sq = 0.0f;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int q = 2 * warp + i;
            float y0 = fmaf(P.w3[0][lane + 32], S.h2[q][lane + 32], P.w3[0][lane] * S.h2[q][lane]);
            float y1 = fmaf(P.w3[1][lane + 32], S.h2[q][lane + 32], P.w3[1][lane] * S.h2[q][lane]);
#pragma unroll
            for (int d = 16; d; d >>= 1) {
                y0 += __shfl_xor_sync(0xFFFFFFFFu, y0, d);
                y1 += __shfl_xor_sync(0xFFFFFFFFu, y1, d);
            }
            const uint32_t sidx = s0 + q;
            if (lane < kOut) {
                float e = 0.0f;
                if (sidx < n) {
                    e = ((lane ? y1 : y0) + P.b3[lane]) - S.ty[q][lane];
                    sq = fmaf(e, e, sq);
                }
                // d(mean squared error)/dy with scale = 1 / (samples * outputs)
                S.dy[q][lane] = 2.0f * scale * e;
            }
        }
        sq += __shfl_xor_sync(0xFFFFFFFFu, sq, 1);
        if (lane == 0) atomicAdd(loss_sum, (double)sq);
        __syncwarp();
        // dL/da2
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int q = 2 * warp + i;
            const float g0 = S.dy[q][0], g1 = S.dy[q][1];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int j = lane + 32 * h;
                S.d2[q][j] = (P.w3[0][j] * g0 + P.w3[1][j] * g1) * gelu_grad(S.a2[q][j]);
            }
        }
    }
    __syncthreads();
    // dL/da1: four units of a sample a thread
    {
        const int q = tid / 16, k = (tid % 16) * 4;
        float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 4
        for (int j = 0; j < kH; j += 4) {
            const float4 d = *reinterpret_cast<const float4*>(&S.d2[q][j]);
            const float dj[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float4 w = *reinterpret_cast<const float4*>(&P.w2[j + i][k]);
                a.x = fmaf(w.x, dj[i], a.x);
                a.y = fmaf(w.y, dj[i], a.y);
                a.z = fmaf(w.z, dj[i], a.z);
                a.w = fmaf(w.w, dj[i], a.w);
            }
        }
        a.x *= gelu_grad(S.a1[q][k]);
        a.y *= gelu_grad(S.a1[q][k + 1]);
        a.z *= gelu_grad(S.a1[q][k + 2]);
        a.w *= gelu_grad(S.a1[q][k + 3]);
        *reinterpret_cast<float4*>(&S.d1[q][k]) = a;
    }
    // parameter gradients, summed over the CTA's samples.  W2: eight inputs
    // of a unit a thread
    {
        const int j = tid / 8, k = (tid % 8) * 8;
        float g[8] = {};
#pragma unroll 4
        for (int q = 0; q < kSamples; ++q) {
            const float d = S.d2[q][j];
            const float4 u = *reinterpret_cast<const float4*>(&S.h1[q][k]);
            const float4 v = *reinterpret_cast<const float4*>(&S.h1[q][k + 4]);
            g[0] = fmaf(d, u.x, g[0]); g[1] = fmaf(d, u.y, g[1]); g[2] = fmaf(d, u.z, g[2]); g[3] = fmaf(d, u.w, g[3]);
            g[4] = fmaf(d, v.x, g[4]); g[5] = fmaf(d, v.y, g[5]); g[6] = fmaf(d, v.z, g[6]); g[7] = fmaf(d, v.w, g[7]);
        }
        red_add4(grad + oW2 + j * kH + k, g[0], g[1], g[2], g[3]);
        red_add4(grad + oW2 + j * kH + k + 4, g[4], g[5], g[6], g[7]);
    }
    __syncthreads();
    // the others, one a thread and round
    for (int e = tid; e < kParams - kH * kH; e += kGradThreads) {
        float acc = 0.0f;
        int at;
        if (e < oB1) {                       // W1[j][k]
            const int j = e / kIn, k = e % kIn;
            for (int q = 0; q < kSamples; ++q) acc = fmaf(S.d1[q][j], S.xin[q][k], acc);
            at = e;
        } else if (e < oW2) {                // b1
            for (int q = 0; q < kSamples; ++q) acc += S.d1[q][e - oB1];
            at = e;
        } else if (e < oW2 + kH) {           // b2
            for (int q = 0; q < kSamples; ++q) acc += S.d2[q][e - oW2];
            at = oB2 + (e - oW2);
        } else if (e < oW2 + kH + kOut * kH) {   // W3[o][j]
            const int i = e - (oW2 + kH), o = i / kH, j = i % kH;
            for (int q = 0; q < kSamples; ++q) acc = fmaf(S.dy[q][o], S.h2[q][j], acc);
            at = oW3 + i;
        } else {                             // b3
            const int o = e - (oW2 + kH + kOut * kH);
            for (int q = 0; q < kSamples; ++q) acc += S.dy[q][o];
            at = oB3 + o;
        }
        atomicAdd(&grad[at], acc);
    }
    if (!adam) return;
    __threadfence();
    __syncthreads();
    if (tid == 0) {
        S.last = atomicAdd(done, 1u) == gridDim.x - 1u;
        __threadfence();
    }
    __syncthreads();
    if (!S.last) return;
    // (the next step's CTAs wait here, not at the start: among this step's they
    // would crowd its free SMs)
    release_next();
    adam_all<kGradThreads>(A, grad);
    if (tid == 0) *done = 0;
}

__global__ void k_to_bf16(const float* __restrict__ master, __nv_bfloat16* __restrict__ wb) {
    wait_for_stream();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kParams) wb[i] = __float2bfloat16_rn(master[i]);
}

// Shuffle keys for one epoch: a splitmix64 hash of (seed, i).
__global__ void k_perm_keys(uint32_t* __restrict__ keys, uint32_t n, uint64_t seed) {
    wait_for_stream();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint64_t z = seed + 0x9E3779B97F4A7C15ull * (uint64_t)(i + 1);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    keys[i] = (uint32_t)((z ^ (z >> 31)) >> 32);
}

// ------------------------------------------------------------ allotment --
// ceil(exp(y + margin) - 1): a count from a prediction in log(1 + count) units.
SR_DEV uint32_t allot_of(float y, float margin) {
    const float a = ceilf(expm1f(fminf(y + margin, 21.0f)));   // exp(21) < 2^31
    return a > 0.0f ? (uint32_t)a : 0u;
}

// Per path: the allotment (path margins, judged path by path) and the
// path's share of the frame capacity (frame margins), summed per scene and
// over the batch.  tot = frame records, frame draws, allotted records,
// allotted draws; scene_tot[S][2] = frame records, frame draws.
__global__ void k_allot(const float* __restrict__ y, uint32_t n_paths, const uint32_t* __restrict__ path_scene,
                        float4 margins, uint32_t* __restrict__ allot, unsigned long long* __restrict__ scene_tot,
                        unsigned long long* __restrict__ tot) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    unsigned long long v[4] = {0, 0, 0, 0};
    if (p < n_paths) {
        const float yr = y[(size_t)p * kOut], yd = y[(size_t)p * kOut + 1];
        const uint32_t ar = allot_of(yr, margins.x), ad = allot_of(yd, margins.y);
        const uint32_t fr = allot_of(yr, margins.z), fd = allot_of(yd, margins.w);
        allot[2 * (size_t)p] = ar;
        allot[2 * (size_t)p + 1] = ad;
        const uint32_t s = path_scene[p];
        atomicAdd(&scene_tot[2 * (size_t)s], (unsigned long long)fr);
        atomicAdd(&scene_tot[2 * (size_t)s + 1], (unsigned long long)fd);
        v[0] = fr;
        v[1] = fd;
        v[2] = ar;
        v[3] = ad;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
#pragma unroll
        for (int o = 16; o; o >>= 1) v[k] += __shfl_xor_sync(0xFFFFFFFFu, v[k], o);
    }
    if (lane == 0) {
#pragma unroll
        for (int k = 0; k < 4; ++k) atomicAdd(&tot[k], v[k]);
    }
}

// Per path: the exact counts against the allotment.  out[0] paths whose
// records exceed their allotment, out[1] likewise for draw records, out[2]
// and out[3] the exact totals.
__global__ void k_judge(const uint32_t* __restrict__ path_first_curve, uint32_t n_paths,
                        const int32_t* __restrict__ count, const uint32_t* __restrict__ path_draw,
                        const uint32_t* __restrict__ allot, unsigned long long* __restrict__ out) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long over_r = 0, over_d = 0, nr = 0, nd = 0;
    if (p < n_paths) {
        for (uint32_t c = path_first_curve[p]; c < path_first_curve[p + 1]; ++c) nr += (uint32_t)count[c];
        nd = path_draw[p];
        over_r = nr > allot[2 * (size_t)p] ? 1u : 0u;
        over_d = nd > allot[2 * (size_t)p + 1] ? 1u : 0u;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        over_r += __shfl_xor_sync(0xFFFFFFFFu, over_r, o);
        over_d += __shfl_xor_sync(0xFFFFFFFFu, over_d, o);
        nr += __shfl_xor_sync(0xFFFFFFFFu, nr, o);
        nd += __shfl_xor_sync(0xFFFFFFFFu, nd, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&out[0], over_r);
        atomicAdd(&out[1], over_d);
        atomicAdd(&out[2], nr);
        atomicAdd(&out[3], nd);
    }
}

// ------------------------------------------------------------- launches --
void launch_path_features(const GeomArgs& g, const uint32_t* path_first_curve, uint32_t n_paths, float* feats,
                          cudaStream_t st) {
    if (!n_paths) return;
    count_launches(1);
    k_path_features<<<(n_paths + 127) / 128, 128, 0, st>>>(g, path_first_curve, n_paths, feats);
}

void launch_path_labels(const uint32_t* path_first_curve, uint32_t n_paths, const int32_t* count,
                        const uint32_t* path_draw, float* labels, cudaStream_t st) {
    if (!n_paths) return;
    count_launches(1);
    k_path_labels<<<(n_paths + 127) / 128, 128, 0, st>>>(path_first_curve, n_paths, count, path_draw, labels);
}

void launch_mlp_predict(const void* wb, const float* master, const float* norm, const float* x, uint32_t n, float* y,
                        int sm_count, cudaStream_t st) {
    if (!n) return;
    count_launches(1);
    constexpr unsigned per = kPredictThreads / 32 * kWarpPaths;
    unsigned blocks = n / per + (n % per ? 1u : 0u);
    const unsigned cap = (unsigned)kPredictCtas * (unsigned)(sm_count > 0 ? sm_count : 148);   // one wave
    if (blocks > cap) blocks = cap;
    launch_after(k_mlp_predict, blocks, kPredictThreads, 0, st, static_cast<const __nv_bfloat16*>(wb), master, norm, x,
                 n, y);
}

static cudaError_t grad_launch(const void* wb, const float* master, const float* norm, const float* x, const float* t,
                               const uint32_t* idx, uint32_t rows, uint32_t n, float* grad, double* loss_sum,
                               bool adam, const AdamArgs& A, uint32_t* done, cudaStream_t st) {
    static std::atomic<uint32_t> attr{0};
    cudaError_t e = cudaSuccess;
    once_per_device(attr, [&] {
        e = cudaFuncSetAttribute(k_mlp_grad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(GradSmem));
    });
    if (e != cudaSuccess) return e;
    count_launches(1);
    launch_after(k_mlp_grad, (n + kSamples - 1) / kSamples, kGradThreads, sizeof(GradSmem), st,
                 static_cast<const __nv_bfloat16*>(wb), master, norm, x, t, idx, rows, n,
                 1.0f / ((float)n * (float)kOut), grad, loss_sum, adam ? 1 : 0, A, done);
    return cudaGetLastError();
}

cudaError_t launch_mlp_grad(const void* wb, const float* master, const float* norm, const float* x, const float* t,
                            const uint32_t* idx, uint32_t n, float* grad, double* loss_sum, cudaStream_t st) {
    if (!n) return cudaSuccess;
    return grad_launch(wb, master, norm, x, t, idx, n, n, grad, loss_sum, false, AdamArgs{}, nullptr, st);
}

cudaError_t launch_mlp_step(void* wb, float* master, const float* norm, const float* x, const float* t,
                            const uint32_t* idx, uint32_t rows, uint32_t n, float* grad, double* loss_sum, float* m,
                            float* v, float lr, float b1, float b2, float eps, float bc1, float bc2, uint32_t* done,
                            cudaStream_t st) {
    if (!n) return cudaSuccess;
    const AdamArgs A{master, m, v, static_cast<__nv_bfloat16*>(wb), lr, b1, b2, eps, bc1, bc2};
    return grad_launch(wb, master, norm, x, t, idx, rows, n, grad, loss_sum, true, A, done, st);
}

void launch_to_bf16(const float* master, void* wb, cudaStream_t st) {
    count_launches(1);
    launch_after(k_to_bf16, (kParams + 255) / 256, 256, 0, st, master, static_cast<__nv_bfloat16*>(wb));
}

void launch_perm_keys(uint32_t* keys, uint32_t n, uint64_t seed, cudaStream_t st) {
    if (!n) return;
    count_launches(1);
    launch_after(k_perm_keys, (n + 255) / 256, 256, 0, st, keys, n, seed);
}

void launch_allot(const float* y, uint32_t n_paths, const uint32_t* path_scene, const float margins[4],
                  uint32_t* allot, unsigned long long* scene_tot, unsigned long long* tot, cudaStream_t st) {
    if (!n_paths) return;
    count_launches(1);
    const float4 m = make_float4(margins[0], margins[1], margins[2], margins[3]);
    k_allot<<<(n_paths + 255) / 256, 256, 0, st>>>(y, n_paths, path_scene, m, allot, scene_tot, tot);
}

void launch_judge(const uint32_t* path_first_curve, uint32_t n_paths, const int32_t* count, const uint32_t* path_draw,
                  const uint32_t* allot, unsigned long long* out, cudaStream_t st) {
    if (!n_paths) return;
    count_launches(1);
    k_judge<<<(n_paths + 255) / 256, 256, 0, st>>>(path_first_curve, n_paths, count, path_draw, allot, out);
}

}  // namespace sr
