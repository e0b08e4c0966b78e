// pf_sizer.cu - the learned per-path sizer: features, a 12 -> 64 -> 64 -> 2 MLP
// (bf16 weights, fp32 accumulation), and its training kernels (forward, backward, Adam).
//
// The reference sizes its microline and fill buffers by running dice/bin, reading the
// count back and re-running on overflow (pathfinder/core/d3d11/renderer.cpp:540-577,
// 707-724, 834-845).  The sizer predicts, per path, log1p(leaf lines) and log1p(fills)
// from cheap geometric features, so a frame can lay out per-path leaf regions and fill
// capacity before flattening, in one pass; the exact count-then-allocate frame remains
// the fallback when a prediction overflows.
#include <math.h>

#include <algorithm>
#include <atomic>

#include "pf_internal.h"

namespace pfc {

namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ uint32_t global_tid() { return blockIdx.x * blockDim.x + threadIdx.x; }

__device__ __forceinline__ float leg_len(float2 a, float2 b) {
    const float dx = b.x - a.x, dy = b.y - a.y;
    return sqrtf(dx * dx + dy * dy);
}

// absolute turning angle between legs a->b and b->c
__device__ __forceinline__ float turn(float2 a, float2 b, float2 c) {
    const float ux = b.x - a.x, uy = b.y - a.y, vx = c.x - b.x, vy = c.y - b.y;
    const float cr = ux * vy - uy * vx, dt = ux * vx + uy * vy;
    if (cr == 0.0f && dt == 0.0f) return 0.0f;
    return fabsf(atan2f(cr, dt));
}

// Per contour: its point-flag counts, control-polygon length and summed turning angle
// (closed around the contour).  Paths sum them over their contours, so a path of thousands of
// contours (a dashed stroke's outline) costs its warp one strided pass over those sums.  A warp per
// contour, its points over the lanes: a point's turn is an arc tangent and its neighbours' loads (a
// thread per contour of up to 64 points took 74 us on the 12,383 contours of mixed 8,192 paths, now
// 11 us).
__device__ __forceinline__ void point_terms(const Batch &b, uint32_t a, uint32_t n, uint32_t i, float &n_on,
                                            float &n_c0, float &n_c1, float &length, float &turning) {
    const uint8_t f = b.flags[a + i];
    n_on += f == 0;
    n_c0 += f == 1;
    n_c1 += f == 2;
    if (n > 1) {
        const float2 q0 = b.points[a + (i == 0 ? n - 1 : i - 1)], q1 = b.points[a + i],
                     q2 = b.points[a + (i + 1 == n ? 0 : i + 1)];
        length += leg_len(q1, q2);
        turning += turn(q0, q1, q2);
    }
}

__global__ void __launch_bounds__(kThreads) k_contour_features(Batch b, float4 *cf) {
    const uint32_t c = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (c >= b.n_contours) return;
    const uint32_t a = b.contour_point_first[c], n = b.contour_point_first[c + 1] - a;
    float n_on = 0, n_c0 = 0, n_c1 = 0, length = 0, turning = 0;
    for (uint32_t i = lane; i < n; i += 32) point_terms(b, a, n, i, n_on, n_c0, n_c1, length, turning);
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        n_on += __shfl_xor_sync(0xffffffffu, n_on, d);
        n_c0 += __shfl_xor_sync(0xffffffffu, n_c0, d);
        n_c1 += __shfl_xor_sync(0xffffffffu, n_c1, d);
        length += __shfl_xor_sync(0xffffffffu, length, d);
        turning += __shfl_xor_sync(0xffffffffu, turning, d);
    }
    if (lane == 0) {
        cf[2 * (size_t)c] = make_float4(n_on, n_c0, n_c1, length);
        cf[2 * (size_t)c + 1] = make_float4(turning, 0.0f, 0.0f, 0.0f);
    }
}

// One warp per path: features from its contours' sums and its bounds / tile rect (after
// k_paths); they need no segment records, so they are ready before the first host
// synchronisation of a frame:
//   0 segments   1 lines   2 quadratics   3 cubics   4 contours   5 box width   6 box height
//   7 box area   8 control-polygon length   9 summed turning angle   10 tiles in the rect
//   11 even-odd flag
// (log1p of every count / length; the reference's outlines are already in canvas space, so
// the transform-scale feature is replaced by the tile count of the clipped rect).
__global__ void k_features(Batch b, const uint2 *path_contours, const float4 *cf, float *feat) {
    const uint32_t p = global_tid() >> 5;
    const int lane = threadIdx.x & 31;
    if (p >= b.n_paths) return;
    const uint2 cr = path_contours[p];
    float n_on = 0, n_c0 = 0, n_c1 = 0, length = 0, turning = 0;
    for (uint32_t c = cr.x + lane; c < cr.y; c += 32) {
        const float4 u = cf[2 * (size_t)c], v = cf[2 * (size_t)c + 1];
        n_on += u.x;
        n_c0 += u.y;
        n_c1 += u.z;
        length += u.w;
        turning += v.x;
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        n_on += __shfl_xor_sync(0xffffffffu, n_on, d);
        n_c0 += __shfl_xor_sync(0xffffffffu, n_c0, d);
        n_c1 += __shfl_xor_sync(0xffffffffu, n_c1, d);
        length += __shfl_xor_sync(0xffffffffu, length, d);
        turning += __shfl_xor_sync(0xffffffffu, turning, d);
    }
    if (lane != 0) return;
    const float4 bb = b.path_bounds[p];
    const float w = fmaxf(bb.z - bb.x, 0.0f), h = fmaxf(bb.w - bb.y, 0.0f);
    const PathDev P = b.paths[p];
    const float tiles = (float)max(P.rx1 - P.rx0, 0) * (float)max(P.ry1 - P.ry0, 0);
    const float n_cubic = n_c1, n_quad = fmaxf(n_c0 - n_c1, 0.0f), n_line = fmaxf(n_on - n_c0, 0.0f);
    float *f = feat + (size_t)p * kSizerIn;
    f[0] = log1pf(n_on);
    f[1] = log1pf(n_line);
    f[2] = log1pf(n_quad);
    f[3] = log1pf(n_cubic);
    f[4] = log1pf((float)(cr.y - cr.x));
    f[5] = log1pf(w);
    f[6] = log1pf(h);
    f[7] = log1pf(w * h);
    f[8] = log1pf(length);
    f[9] = log1pf(turning);
    f[10] = log1pf(tiles);
    f[11] = (P.flags & 1u) ? 1.0f : 0.0f;
}

// Per-path leaf budget (and fill estimate) from the sizer's prediction:
// budget = ceil(expm1(prediction) * mul + add), and at least the path's segment count: every
// segment yields at least one leaf, and a segment's first leaf goes to the slot of its own
// index in the path's region (k_flatten_pool), so the region's write cursor starts past them.
__global__ void k_budgets(Batch b, const float *pred, float mul, float add, uint32_t *leaf_budget,
                          uint32_t *fill_budget, uint32_t *leaf_cursor) {
    const uint32_t p = global_tid();
    if (p >= b.n_paths) return;
    const float l = fmaxf(expm1f(fminf(pred[2 * p + 0], 30.0f)), 0.0f);
    const float f = fmaxf(expm1f(fminf(pred[2 * p + 1], 30.0f)), 0.0f);
    const uint2 cr = b.path_contours[p];
    const uint32_t n_segs = b.contour_segs[cr.y] - b.contour_segs[cr.x];
    leaf_budget[p] = max((uint32_t)fminf(ceilf(l * mul + add), 1.0e9f), n_segs);
    fill_budget[p] = (uint32_t)fminf(ceilf(f * mul + add), 1.0e9f);
    leaf_cursor[p] = n_segs;
}

// Exact per-path counts of the last exact frame (training labels): leaf lines and fills.
__global__ void k_path_counts(Batch b, const uint2 *path_contours, uint32_t *leaves, uint32_t *fills) {
    const uint32_t p = global_tid();
    if (p >= b.n_paths) return;
    const uint2 cr = path_contours[p];
    const uint32_t s0 = b.contour_segs[cr.x], s1 = b.contour_segs[cr.y];
    leaves[p] = b.seg_leaves[s1] - b.seg_leaves[s0];
    const uint32_t t0 = b.path_tiles[p], t1 = b.path_tiles[p + 1];
    fills[p] = t1 > t0 ? b.tile_fills[t1 - 1] - b.path_fill[p] : 0u;
}

// ---------------------------------------------------------------------------
// MLP.  Parameter block layout (floats): W1[64][12] b1[64] W2[64][64] b2[64] W3[2][64] b3[2].

constexpr int kH = kSizerHidden, kI = kSizerIn, kO = kSizerOut;
constexpr int kOffW1 = 0, kOffB1 = kOffW1 + kH * kI, kOffW2 = kOffB1 + kH, kOffB2 = kOffW2 + kH * kH,
              kOffW3 = kOffB2 + kH, kOffB3 = kOffW3 + kO * kH, kParams = kOffB3 + kO;
static_assert(kParams == kSizerParams, "parameter count");

// Weights are stored and used in bf16; activations and accumulation are fp32, so the contractions run
// on the fp32 pipes: 14,000 multiply-adds a sample in training, 5,000 in prediction.  What bounds
// them is how many operands each needs from shared memory, so a block works on kTile samples at a
// time with a tile of 8 x 4 results per thread (12 16-byte reads per 128 multiply-adds), all
// activations in shared memory, sample by sample.  Blocks stay on their SM (three fit) and take tiles
// in turn, so the weight gradients stay in registers until the end: one atomic per block and
// parameter.  (A sample per thread, weights read one by one, and the gradients of 64 samples added
// with 5,122 atomics each: 65,536 samples trained in 298 us, predicted in 108 us; now 88 and
// 35 us.)
constexpr int kMlpThreads = 128, kMlpTile = 64, kMlpBlocks = 3;  // blocks per SM
static_assert(kMlpThreads == kO * kH && kOffW2 % 8 == 0, "the weights' loads");
constexpr int kPad = kH + 4;  // row of a sample's activations: 16-byte aligned, rows in other banks

struct MlpShared {
    float w1t[kI][kH];   // [k][i]
    float w2t[kH][kH];   // [k][i]
    float w2[kH][kH];    // [i][k]
    float w3[kO][kH];
    float b1[kH], b2[kH], b3[4];
    float x[kMlpTile][kI];
    float h1[kMlpTile][kPad];  // then dL/d(pre-activation 1)
    float h2[kMlpTile][kPad];  // then dL/d(pre-activation 2)
    float dy[kMlpTile][kO];
};

// acc[j][i] += sum over k of w[k][o + i] * act[s + j][k], for this thread's 8 outputs and 4 samples
template <int kK, int kStride>
__device__ __forceinline__ void mlp_gemm(const float (*w)[kH], const float *act, int o, int s, float acc[4][8]) {
#pragma unroll 4
    for (int k = 0; k < kK; k += 4) {
        float4 v[4];
#pragma unroll
        for (int j = 0; j < 4; j++) v[j] = *reinterpret_cast<const float4 *>(act + (s + j) * kStride + k);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const float4 u0 = *reinterpret_cast<const float4 *>(&w[k + q][o]);
            const float4 u1 = *reinterpret_cast<const float4 *>(&w[k + q][o + 4]);
            const float u[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float a = q == 0 ? v[j].x : q == 1 ? v[j].y : q == 2 ? v[j].z : v[j].w;
#pragma unroll
                for (int i = 0; i < 8; i++) acc[j][i] = fmaf(u[i], a, acc[j][i]);
            }
        }
    }
}

__device__ __forceinline__ void mlp_store(float (*dst)[kPad], int o, int s, const float v[4][8]) {
#pragma unroll
    for (int j = 0; j < 4; j++) {
        *reinterpret_cast<float4 *>(&dst[s + j][o]) = make_float4(v[j][0], v[j][1], v[j][2], v[j][3]);
        *reinterpret_cast<float4 *>(&dst[s + j][o + 4]) = make_float4(v[j][4], v[j][5], v[j][6], v[j][7]);
    }
}

// kTrain false: predictions into out.  kTrain true: forward and backward of the mini-batch, weight
// gradients added to grad and squared errors to loss (mean over samples and outputs of (y - t)^2
// once the caller divides).  Samples past n have zero features and no error.
template <bool kTrain>
__global__ void __launch_bounds__(kMlpThreads, kMlpBlocks) k_mlp(const __nv_bfloat16 *w, const float *feat,
                                                        const float *target, const uint32_t *index, uint32_t n,
                                                        float inv_count, float *out, float *grad, float *loss) {
    extern __shared__ float4 smem[];
    MlpShared &S = *reinterpret_cast<MlpShared *>(smem);
    const int t = threadIdx.x;
    // the weights, read eight (W2) or two (W1) at a time along k and stored along i
    const uint32_t *const pairs = reinterpret_cast<const uint32_t *>(w);
    auto low = [](uint32_t v) { return __uint_as_float(v << 16); };  // bf16 to fp32
    auto high = [](uint32_t v) { return __uint_as_float(v & 0xffff0000u); };
#pragma unroll
    for (int q = t; q < kH * kI / 2; q += kMlpThreads) {
        const int i = q % kH, k = q / kH * 2;
        const uint32_t v = pairs[(kOffW1 + i * kI + k) / 2];
        S.w1t[k][i] = low(v);
        S.w1t[k + 1][i] = high(v);
    }
#pragma unroll
    for (int q = t; q < kH * kH / 8; q += kMlpThreads) {
        const int i = q % kH, k = q / kH * 8;
        const uint4 v = *reinterpret_cast<const uint4 *>(pairs + (kOffW2 + i * kH + k) / 2);
        const float f[8] = {low(v.x), high(v.x), low(v.y), high(v.y), low(v.z), high(v.z), low(v.w), high(v.w)};
#pragma unroll
        for (int j = 0; j < 8; j++) S.w2t[k + j][i] = f[j];
        if (kTrain) {
            *reinterpret_cast<float4 *>(&S.w2[i][k]) = make_float4(f[0], f[1], f[2], f[3]);
            *reinterpret_cast<float4 *>(&S.w2[i][k + 4]) = make_float4(f[4], f[5], f[6], f[7]);
        }
    }
    S.w3[t / kH][t % kH] = __bfloat162float(w[kOffW3 + t]);
    if (t < kH) {
        S.b1[t] = __bfloat162float(w[kOffB1 + t]);
        S.b2[t] = __bfloat162float(w[kOffB2 + t]);
    }
    if (t < kO) S.b3[t] = __bfloat162float(w[kOffB3 + t]);
    const int o = (t & 7) * 8, s = (t >> 3) * 4;            // this thread's outputs and samples of a layer
    const int gi = (t >> 4) * 8, gk = (t & 15) * 4;         // its part of W2's gradient
    const int xi = t >> 1, xk = (t & 1) * 6;                // of W1's
    float g2[8][4] = {}, g1[6] = {}, g3 = 0.0f, gb = 0.0f, gb3 = 0.0f, err = 0.0f;
    const uint32_t tiles = (n + kMlpTile - 1) / kMlpTile;
    for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        __syncthreads();
        for (int q = t; q < kMlpTile * kI; q += kMlpThreads) {
            const uint32_t j = tile * kMlpTile + q / kI;
            float v = 0.0f;
            if (j < n) v = feat[(size_t)(kTrain && index ? index[j] : j) * kI + q % kI];
            S.x[q / kI][q % kI] = v;
        }
        __syncthreads();
        float acc[4][8];
        auto layer = [&](const float *bias) {
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const float v = bias ? bias[o + i] : 0.0f;
#pragma unroll
                for (int j = 0; j < 4; j++) acc[j][i] = v;
            }
        };
        auto relu = [&]() {
#pragma unroll
            for (int j = 0; j < 4; j++)
#pragma unroll
                for (int i = 0; i < 8; i++) acc[j][i] = fmaxf(acc[j][i], 0.0f);
        };
        layer(S.b1);
        mlp_gemm<kI, kI>(S.w1t, &S.x[0][0], o, s, acc);
        relu();
        mlp_store(S.h1, o, s, acc);
        __syncthreads();
        layer(S.b2);
        mlp_gemm<kH, kPad>(S.w2t, &S.h1[0][0], o, s, acc);
        relu();
        mlp_store(S.h2, o, s, acc);
        __syncthreads();
        {
            // the outputs: a sample and output per thread
            const int m = t >> 1, c = t & 1;
            float y = S.b3[c];
#pragma unroll
            for (int k = 0; k < kH; k += 4) {
                const float4 h = *reinterpret_cast<const float4 *>(&S.h2[m][k]);
                const float4 u = *reinterpret_cast<const float4 *>(&S.w3[c][k]);
                y = fmaf(u.x, h.x, fmaf(u.y, h.y, fmaf(u.z, h.z, fmaf(u.w, h.w, y))));
            }
            const uint32_t j = tile * kMlpTile + m;
            if (!kTrain) {
                if (j < n) out[(size_t)j * kO + c] = y;
            } else {
                const float e = j < n ? y - target[(size_t)(index ? index[j] : j) * kO + c] : 0.0f;
                err = fmaf(e, e, err);
                S.dy[m][c] = 2.0f * e * inv_count;
            }
        }
        if constexpr (kTrain) {
            __syncthreads();
            // layer 3's gradient: a weight per thread (and the biases by the threads of weight 0)
            {
                const int c = t >> 6, k = t & 63;
#pragma unroll 8
                for (int m = 0; m < kMlpTile; m++) {
                    g3 = fmaf(S.dy[m][c], S.h2[m][k], g3);
                    gb3 += S.dy[m][c];
                }
            }
            __syncthreads();
            // back through layer 3 and the ReLU of layer 2, in place of its activations
#pragma unroll
            for (int j = 0; j < 4; j++)
#pragma unroll
                for (int i = 0; i < 8; i++)
                    acc[j][i] = acc[j][i] > 0.0f ? fmaf(S.w3[0][o + i], S.dy[s + j][0], S.w3[1][o + i] * S.dy[s + j][1]) : 0.0f;
            mlp_store(S.h2, o, s, acc);
            __syncthreads();
            // layer 2's gradient
#pragma unroll 4
            for (int m = 0; m < kMlpTile; m++) {
                const float4 d0 = *reinterpret_cast<const float4 *>(&S.h2[m][gi]);
                const float4 d1 = *reinterpret_cast<const float4 *>(&S.h2[m][gi + 4]);
                const float4 h = *reinterpret_cast<const float4 *>(&S.h1[m][gk]);
                const float d[8] = {d0.x, d0.y, d0.z, d0.w, d1.x, d1.y, d1.z, d1.w};
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    g2[i][0] = fmaf(d[i], h.x, g2[i][0]);
                    g2[i][1] = fmaf(d[i], h.y, g2[i][1]);
                    g2[i][2] = fmaf(d[i], h.z, g2[i][2]);
                    g2[i][3] = fmaf(d[i], h.w, g2[i][3]);
                }
            }
            // back through layer 2 and the ReLU of layer 1
            layer(nullptr);
            mlp_gemm<kH, kPad>(S.w2, &S.h2[0][0], o, s, acc);
#pragma unroll
            for (int j = 0; j < 4; j++)
#pragma unroll
                for (int i = 0; i < 8; i++) acc[j][i] = S.h1[s + j][o + i] > 0.0f ? acc[j][i] : 0.0f;
            __syncthreads();  // every thread has read layer 1's activations
            mlp_store(S.h1, o, s, acc);
            __syncthreads();
            // layer 1's gradient, and the biases of layers 2 (threads 0-63) and 1
            const float (*const bias_rows)[kPad] = t < kH ? S.h2 : S.h1;
#pragma unroll 4
            for (int m = 0; m < kMlpTile; m++) {
                const float d = S.h1[m][xi];
#pragma unroll
                for (int k = 0; k < 6; k++) g1[k] = fmaf(d, S.x[m][xk + k], g1[k]);
                gb += bias_rows[m][t & 63];
            }
        }
    }
    if constexpr (kTrain) {
#pragma unroll
        for (int i = 0; i < 8; i++)
#pragma unroll
            for (int k = 0; k < 4; k++) atomicAdd(&grad[kOffW2 + (gi + i) * kH + gk + k], g2[i][k]);
#pragma unroll
        for (int k = 0; k < 6; k++) atomicAdd(&grad[kOffW1 + xi * kI + xk + k], g1[k]);
        atomicAdd(&grad[kOffW3 + t], g3);
        atomicAdd(&grad[(t < kH ? kOffB2 : kOffB1) + (t & 63)], gb);
        if ((t & 63) == 0) atomicAdd(&grad[kOffB3 + (t >> 6)], gb3);
        for (int d = 16; d > 0; d >>= 1) err += __shfl_xor_sync(0xffffffffu, err, d);
        // one addition per block: a sum of a quarter of the terms, and so fewer roundings
        __syncthreads();
        if ((t & 31) == 0) S.b3[t >> 5] = err;
        __syncthreads();
        if (t == 0) atomicAdd(loss, (S.b3[0] + S.b3[1]) + (S.b3[2] + S.b3[3]));
    }
}

// Training step, part 2: Adam on fp32 master weights, bf16 copy for the next forward.
__global__ void k_adam(float *master, __nv_bfloat16 *w, float *grad, float *m, float *v, float lr, float beta1,
                       float beta2, float eps, float bc1, float bc2) {
    const int q = global_tid();
    if (q >= kParams) return;
    const float g = grad[q];
    const float mq = beta1 * m[q] + (1.0f - beta1) * g;
    const float vq = beta2 * v[q] + (1.0f - beta2) * g * g;
    m[q] = mq;
    v[q] = vq;
    const float upd = lr * (mq / bc1) / (sqrtf(vq / bc2) + eps);
    const float nw = master[q] - upd;
    master[q] = nw;
    w[q] = __float2bfloat16_rn(nw);
    grad[q] = 0.0f;
}

}  // namespace

cudaError_t launch_features(const Batch &b, const uint2 *path_contours, float4 *contour_scratch, float *feat,
                            cudaStream_t st) {
    if (b.n_paths) {
        if (b.n_contours) {
            k_contour_features<<<(b.n_contours + kThreads / 32 - 1) / (kThreads / 32), kThreads, 0, st>>>(b, contour_scratch);
            count_launches(1);
        }
        k_features<<<(unsigned)((uint64_t(b.n_paths) * 32 + kThreads - 1) / kThreads), kThreads, 0, st>>>(
            b, path_contours, contour_scratch, feat);
        count_launches(1);
    }
    return cudaGetLastError();
}

cudaError_t launch_budgets(const Batch &b, const float *pred, float mul, float add, uint32_t *leaf_budget,
                           uint32_t *fill_budget, uint32_t *leaf_cursor, cudaStream_t st) {
    if (b.n_paths) {
        k_budgets<<<(b.n_paths + kThreads - 1) / kThreads, kThreads, 0, st>>>(b, pred, mul, add, leaf_budget,
                                                                             fill_budget, leaf_cursor);
        count_launches(1);
    }
    return cudaGetLastError();
}

cudaError_t launch_path_counts(const Batch &b, const uint2 *path_contours, uint32_t *leaves, uint32_t *fills,
                               cudaStream_t st) {
    if (b.n_paths) {
        k_path_counts<<<(b.n_paths + kThreads - 1) / kThreads, kThreads, 0, st>>>(b, path_contours, leaves, fills);
        count_launches(1);
    }
    return cudaGetLastError();
}

// As many blocks as the SMs hold, no more than there are tiles of samples.
template <bool kTrain>
static cudaError_t launch_mlp(const __nv_bfloat16 *w, const float *feat, const float *target, const uint32_t *index,
                              uint32_t n, float *out, float *grad, float *loss, cudaStream_t st) {
    if (!n) return cudaSuccess;
    static std::atomic<uint64_t> configured{0};  // devices the kernel's shared memory is set up on
    int dev = 0, sms = 152;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess && !(dev < 64 && (configured.load() >> dev & 1u))) {
        e = cudaFuncSetAttribute(k_mlp<kTrain>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(MlpShared));
        if (e == cudaSuccess && dev < 64) configured.fetch_or(uint64_t(1) << dev);
    }
    if (e != cudaSuccess) return e;
    const unsigned tiles = (unsigned)((uint64_t(n) + kMlpTile - 1) / kMlpTile);
    k_mlp<kTrain><<<std::min(tiles, (unsigned)kMlpBlocks * (unsigned)sms), kMlpThreads, sizeof(MlpShared), st>>>(
        w, feat, target, index, n, 1.0f / ((float)n * kO), out, grad, loss);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_mlp_predict(const __nv_bfloat16 *w, const float *feat, uint32_t n, float *out, cudaStream_t st) {
    return launch_mlp<false>(w, feat, nullptr, nullptr, n, out, nullptr, nullptr, st);
}

cudaError_t launch_mlp_grad(const __nv_bfloat16 *w, const float *feat, const float *target, const uint32_t *index,
                            uint32_t n, float *grad, float *loss, cudaStream_t st) {
    return launch_mlp<true>(w, feat, target, index, n, nullptr, grad, loss, st);
}

cudaError_t launch_adam(float *master, __nv_bfloat16 *w, float *grad, float *m, float *v, float lr, int step,
                        cudaStream_t st) {
    const float b1 = 0.9f, b2 = 0.999f;
    const float bc1 = 1.0f - powf(b1, (float)step), bc2 = 1.0f - powf(b2, (float)step);
    k_adam<<<(kParams + 255) / 256, 256, 0, st>>>(master, w, grad, m, v, lr, b1, b2, 1e-8f, bc1, bc2);
    count_launches(1);
    return cudaGetLastError();
}

}  // namespace pfc
