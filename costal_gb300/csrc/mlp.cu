// The learned block-pruning model: features, forward, backward, Adam (all hand-written CUDA).
//
// Input of row i: its normalised coordinates (d values) and its 64 largest cosines to the 256
// k-means centroids, sorted descending (the "distances to the 64 nearest centroids"). Network:
// F = d + 64 → 128 (ReLU) → 128 (ReLU) → 1 (linear), predicting the row's k-th-neighbour cosine.
// Training (costal_mlp_train) uses the pinball loss at a low quantile, so the prediction sits below
// the true k-th score for most rows: it only sets a skip threshold, and every skip is certified
// after the fact (a query whose k-th score does not beat its skipped blocks' bound is rescanned).
// Training runs the FP32 forward of that definition; inference runs on the tensor cores with bf16
// operands (weights, features and first-layer activations) and FP32 accumulation. Gradients are
// summed over fixed 32-row groups and then over the groups in order, so training is deterministic.

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include "common.cuh"
#include "mlp.h"

namespace costal {
namespace mlp {

constexpr int R = 32;  // rows of a gradient group (one CTA)

struct Off {
    size_t w1, b1, w2, b2, w3, b3;
};
__host__ __device__ inline Off offsets(int F) {
    Off o;
    o.w1 = 0;
    o.b1 = o.w1 + (size_t)MLP_H * F;
    o.w2 = o.b1 + MLP_H;
    o.b2 = o.w2 + (size_t)MLP_H * MLP_H;
    o.w3 = o.b2 + MLP_H;
    o.b3 = o.w3 + MLP_H;
    return o;
}

// ---- features ---------------------------------------------------------------------------------
// One warp per row (two rows at a time, interleaved): the row's (at most 64) coordinates loaded once, two per lane, and broadcast by
// shuffles; lane L takes the 8 consecutive centroids 8L … 8L + 7, read as two 16-byte words per
// dimension from a transposed shared copy laid out so that a warp's words are contiguous (no bank
// conflicts); then a branch-free warp bitonic sort of the 256 cosines (descending; only the values
// are kept, so ties need no order) in which strides below 8 stay in a lane's registers, and the first
// 64 (lanes 0-7) are kept. Each cosine is the same FMA chain over the dimensions in order.

// Bitonic sort of R warp-distributed arrays at once (independent sorts interleaved stage by stage, so
// that each stage's shuffles and compare-exchanges of one array hide the latencies of the other's),
// lane-major (position p = 8·lane + s), descending.
template <int R>
__device__ __forceinline__ void warp_sort_desc_lane8(float (&v)[R][8], int lane) {
#pragma unroll
    for (int size = 2; size <= 256; size <<= 1) {
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            if (stride < 8) {
#pragma unroll
                for (int s = 0; s < 8; ++s) {
                    const int t = s ^ stride;
                    if (t > s) {
                        const bool desc = ((8 * lane + s) & size) == 0;
#pragma unroll
                        for (int r = 0; r < R; ++r) {
                            const float hi = fmaxf(v[r][s], v[r][t]), lo = fminf(v[r][s], v[r][t]);
                            v[r][s] = desc ? hi : lo;
                            v[r][t] = desc ? lo : hi;
                        }
                    }
                }
            } else {
#pragma unroll
                for (int s = 0; s < 8; ++s) {
                    const int p = 8 * lane + s;
                    const bool keep_max = ((p & stride) == 0) == ((p & size) == 0);
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const float o = __shfl_xor_sync(COSTAL_FULL_MASK, v[r][s], stride >> 3);
                        v[r][s] = keep_max ? fmaxf(v[r][s], o) : fminf(v[r][s], o);
                    }
                }
            }
        }
    }
}

constexpr int FEAT_C = 256;  // centroid slots of the feature kernel (K ≤ 256)

__global__ void k_features(const float* __restrict__ xsT, int np, int d, const float* __restrict__ cent, int K,
                           const uint32_t* __restrict__ rows, int m, float* __restrict__ feat) {
    // [d][256]: for dimension t, word h (0, 1) of lane L sits at t·256 + 128·h + 4·L, holding centroids
    // 8L + 4h … 8L + 4h + 3 (zero past K)
    extern __shared__ float4 c_s4[];
    float* c_s = reinterpret_cast<float*>(c_s4);
    for (int e = threadIdx.x; e < d * FEAT_C; e += blockDim.x) {
        const int t = e / FEAT_C, q = e % FEAT_C;
        const int h = q >> 7, L = (q & 127) >> 2, j = q & 3;
        const int c = 8 * L + 4 * h + j;
        c_s[e] = c < K ? cent[(size_t)c * d + t] : 0.0f;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int F = d + MLP_TOPC;
    const int wpb = blockDim.x >> 5;
    // grid-stride over pairs of rows, one warp per pair (the two rows' chains interleave): the
    // centroids are loaded once per CTA. A pair's second row past m repeats the first and is not stored.
    constexpr int R2 = 2;
    const int stride = gridDim.x * wpb;
    for (int i0 = blockIdx.x * wpb + (threadIdx.x >> 5); i0 < m; i0 += R2 * stride) {
        int ii[R2];
        float x0[R2], x1[R2], dot[R2][8];
#pragma unroll
        for (int q = 0; q < R2; ++q) {
            ii[q] = i0 + q * stride;
            const int i = ii[q] < m ? ii[q] : i0;
            const uint32_t r = rows ? rows[i] : (uint32_t)i;
            x0[q] = lane < d ? xsT[(size_t)lane * np + r] : 0.0f;
            x1[q] = lane + 32 < d ? xsT[(size_t)(lane + 32) * np + r] : 0.0f;
#pragma unroll
            for (int s = 0; s < 8; ++s) dot[q][s] = 0.0f;
        }
        for (int t = 0; t < d; ++t) {
            const float4 w0 = c_s4[t * (FEAT_C / 4) + lane], w1 = c_s4[t * (FEAT_C / 4) + 32 + lane];
#pragma unroll
            for (int q = 0; q < R2; ++q) {
                const float a = __shfl_sync(COSTAL_FULL_MASK, t < 32 ? x0[q] : x1[q], t & 31);
                dot[q][0] = fmaf(a, w0.x, dot[q][0]);
                dot[q][1] = fmaf(a, w0.y, dot[q][1]);
                dot[q][2] = fmaf(a, w0.z, dot[q][2]);
                dot[q][3] = fmaf(a, w0.w, dot[q][3]);
                dot[q][4] = fmaf(a, w1.x, dot[q][4]);
                dot[q][5] = fmaf(a, w1.y, dot[q][5]);
                dot[q][6] = fmaf(a, w1.z, dot[q][6]);
                dot[q][7] = fmaf(a, w1.w, dot[q][7]);
            }
        }
#pragma unroll
        for (int q = 0; q < R2; ++q)
#pragma unroll
            for (int s = 0; s < 8; ++s)
                if (8 * lane + s >= K) dot[q][s] = -CUDART_INF_F;
        warp_sort_desc_lane8<R2>(dot, lane);
#pragma unroll
        for (int q = 0; q < R2; ++q) {
            if (ii[q] >= m) continue;
            float* f = feat + (size_t)ii[q] * F;
            if (lane < d) f[lane] = x0[q];
            if (lane + 32 < d) f[lane + 32] = x1[q];
            if (lane < MLP_TOPC / 8) {
#pragma unroll
                for (int s = 0; s < 8; ++s) f[d + 8 * lane + s] = dot[q][s];
            }
        }
    }
}

// ---- inference ----------------------------------------------------------------------------------
// On the tensor cores (mma.sync m16n8k16, bf16 operands, FP32 accumulation): the weights, rounded to
// bf16, stay in shared memory ([unit][input], which is the MMA's column-major B) while persistent CTAs
// of 8 warps walk 128-row tiles, 16 rows a warp. Layer 1 multiplies the tile's features (rounded to
// bf16, row-major A in shared memory) by W1ᵀ into 16 accumulator fragments of 8 units; bias and ReLU
// are applied in registers, and the fragments, rounded to bf16, are layer 2's A operand as they stand
// (the accumulator layout of two adjacent 8-unit tiles is the A layout of one 16-wide K step), so the
// activations never leave the registers. Layer 2 likewise; the output is the dot of ReLU(layer 2) with
// w3 in FP32: each thread's 32 units, then the four threads of a row in a fixed tree, plus b3.
// Padded inputs (K up to the next multiple of 16) and rows past m are zero.
constexpr int IR = 128;           // rows per tile
constexpr int IT = 256;           // threads (8 warps × 16 rows)
constexpr int IKP = MLP_MAXF + 8;  // shared-memory row stride (bf16) of W1 and the features: conflict-free
constexpr int IHP = MLP_H + 8;     // row stride of W2

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);  // .x = lo (low half), .y = hi
    return *reinterpret_cast<const uint32_t*>(&v);
}

__device__ __forceinline__ void mma_bf16_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__global__ void __launch_bounds__(IT) k_infer(const float* __restrict__ P, int F, const float* __restrict__ feat,
                                              int m, float* __restrict__ out) {
    extern __shared__ __align__(16) unsigned char smem_i[];
    __nv_bfloat16* w1s = reinterpret_cast<__nv_bfloat16*>(smem_i);  // [H][IKP]
    __nv_bfloat16* w2s = w1s + (size_t)MLP_H * IKP;                  // [H][IHP]
    __nv_bfloat16* xs = w2s + (size_t)MLP_H * IHP;                   // [IR][IKP] the tile's features
    float* b1 = reinterpret_cast<float*>(xs + (size_t)IR * IKP);     // [H]
    float* b2 = b1 + MLP_H;                                          // [H]
    float* w3 = b2 + MLP_H;                                          // [H]
    const Off o = offsets(F);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, tq = lane & 3;  // the fragment's row group and thread in group
    const int KS1 = (F + 15) >> 4;           // layer-1 K steps
    const int kp = KS1 * 16;
    for (int e = tid; e < MLP_H * kp; e += IT) {
        const int u = e / kp, t = e - u * kp;
        w1s[u * IKP + t] = __float2bfloat16_rn(t < F ? P[o.w1 + (size_t)u * F + t] : 0.0f);
    }
    for (int e = tid; e < MLP_H * MLP_H; e += IT) {
        const int u = e / MLP_H, t = e - u * MLP_H;
        w2s[u * IHP + t] = __float2bfloat16_rn(P[o.w2 + e]);
    }
    if (tid < MLP_H) {
        b1[tid] = P[o.b1 + tid];
        b2[tid] = P[o.b2 + tid];
        w3[tid] = P[o.w3 + tid];
    }
    const float b3 = P[o.b3];
    const int ntiles = (m + IR - 1) / IR;
    const int r_w = warp * 16;  // the warp's first row in the tile
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int r0 = tile * IR;
        __syncthreads();  // the previous tile's readers of xs are done (and the weights loaded)
        for (int e = tid; e < IR * kp; e += IT) {
            const int r = e / kp, t = e - r * kp;
            xs[r * IKP + t] = __float2bfloat16_rn(r0 + r < m && t < F ? feat[(size_t)(r0 + r) * F + t] : 0.0f);
        }
        __syncthreads();
        // layer 1: acc[j] = the 16 rows × units 8j … 8j+7
        float acc[16][4];
#pragma unroll
        for (int j = 0; j < 16; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0f;
        for (int ks = 0; ks < KS1; ++ks) {
            const int k0 = ks * 16 + 2 * tq;
            uint32_t a[4];
            a[0] = *reinterpret_cast<const uint32_t*>(xs + (r_w + g) * IKP + k0);
            a[1] = *reinterpret_cast<const uint32_t*>(xs + (r_w + g + 8) * IKP + k0);
            a[2] = *reinterpret_cast<const uint32_t*>(xs + (r_w + g) * IKP + k0 + 8);
            a[3] = *reinterpret_cast<const uint32_t*>(xs + (r_w + g + 8) * IKP + k0 + 8);
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const __nv_bfloat16* wr = w1s + (8 * j + g) * IKP + k0;
                mma_bf16_16816(acc[j], a, *reinterpret_cast<const uint32_t*>(wr),
                               *reinterpret_cast<const uint32_t*>(wr + 8));
            }
        }
        // bias + ReLU, rounded to bf16: layer 2's A fragments (K step s = units 16s … 16s+15)
        uint32_t h[8][4];
#pragma unroll
        for (int s2 = 0; s2 < 8; ++s2) {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int j = 2 * s2 + half, u = 8 * j + 2 * tq;
                const float bu = b1[u], bv = b1[u + 1];
                h[s2][2 * half] = pack_bf16(fmaxf(acc[j][0] + bu, 0.0f), fmaxf(acc[j][1] + bv, 0.0f));
                h[s2][2 * half + 1] = pack_bf16(fmaxf(acc[j][2] + bu, 0.0f), fmaxf(acc[j][3] + bv, 0.0f));
            }
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0f;
#pragma unroll
        for (int s2 = 0; s2 < 8; ++s2) {
            // A fragment order: (row g, k lo), (row g + 8, k lo), (row g, k hi), (row g + 8, k hi)
            const uint32_t a[4] = {h[s2][0], h[s2][1], h[s2][2], h[s2][3]};
            const int k0 = s2 * 16 + 2 * tq;
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const __nv_bfloat16* wr = w2s + (8 * j + g) * IHP + k0;
                mma_bf16_16816(acc[j], a, *reinterpret_cast<const uint32_t*>(wr),
                               *reinterpret_cast<const uint32_t*>(wr + 8));
            }
        }
        // output: Σ_u w3[u]·ReLU(layer 2 + b2) for rows g and g + 8, units 8j + 2tq, 8j + 2tq + 1
        float pg = 0.0f, pg8 = 0.0f;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const int u = 8 * j + 2 * tq;
            pg = fmaf(w3[u], fmaxf(acc[j][0] + b2[u], 0.0f), pg);
            pg = fmaf(w3[u + 1], fmaxf(acc[j][1] + b2[u + 1], 0.0f), pg);
            pg8 = fmaf(w3[u], fmaxf(acc[j][2] + b2[u], 0.0f), pg8);
            pg8 = fmaf(w3[u + 1], fmaxf(acc[j][3] + b2[u + 1], 0.0f), pg8);
        }
#pragma unroll
        for (int off = 1; off < 4; off <<= 1) {
            pg += __shfl_xor_sync(COSTAL_FULL_MASK, pg, off);
            pg8 += __shfl_xor_sync(COSTAL_FULL_MASK, pg8, off);
        }
        if (tq == 0) {
            const int r = r0 + r_w + g;
            if (r < m) out[r] = b3 + pg;
            if (r + 8 < m) out[r + 8] = b3 + pg8;
        }
    }
}

// ---- training -----------------------------------------------------------------------------------
// Per CTA: the FP32 forward of its 32 rows, the pinball-loss gradient (mean over all m rows), and the
// gradient of every parameter summed over the CTA's rows in row order → partial[blockIdx.x][nparams].
// Every sum is one FMA chain in the order of its index (inputs, units or rows), so a tile's shape does
// not show in the result. Bound by shared-memory loads: both weight matrices and the activations stay
// in shared memory (row strides of 4 × an odd number of words: conflict-free 16-byte loads down a
// column of rows), and a thread keeps 4 rows × 4 units (8 × 4 for the weight gradients), so that an
// operand word serves 4 FMAs. A thread per unit that read its weights' rows from global memory, one
// load an FMA and lanes F words apart, made a step of 2,048 rows (F = 104, 64 CTAs) take 0.447 ms; with
// this form it takes 0.045 (this kernel 0.032, k_adam 0.009). W2 arrives while layer 1 runs.
constexpr int GT = 256;          // threads: 8 warps × 4 rows, lane L's units L, L + 32, L + 64, L + 96
constexpr int GS = MLP_H + 4;    // row stride (words) of W2 and the hidden activations
__host__ __device__ inline int grad_stride(int F) {  // of W1 and the features
    const int q = (F + 3) / 4;
    return 4 * (q | 1);
}

__device__ __forceinline__ void cp4(float* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void cp16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src));
}

// acc[i][c] += Σ_t x[row i][t] · w[unit c][t] in t order (i: 4 rows from x, c: units lane + 32c of w).
__device__ __forceinline__ void layer_tile(float (&acc)[4][4], const float* x, int xs, const float* w, int ws, int n) {
    int t = 0;
#pragma unroll 2
    for (; t + 4 <= n; t += 4) {
        float4 a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(x + i * xs + t);
#pragma unroll
        for (int c = 0; c < 4; ++c) b[c] = *reinterpret_cast<const float4*>(w + 32 * c * ws + t);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                acc[i][c] = fmaf(b[c].x, a[i].x, acc[i][c]);
                acc[i][c] = fmaf(b[c].y, a[i].y, acc[i][c]);
                acc[i][c] = fmaf(b[c].z, a[i].z, acc[i][c]);
                acc[i][c] = fmaf(b[c].w, a[i].w, acc[i][c]);
            }
    }
    for (; t < n; ++t)
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[i][c] = fmaf(w[32 * c * ws + t], x[i * xs + t], acc[i][c]);
}

// G[j][t] = Σ_r dz[r][j] · x[r][t] in row order, for the warp's 16 units j and all t < n.
__device__ __forceinline__ void weight_grad(float* __restrict__ G, const float* dz, const float* x, int xs, int n,
                                            int warp, int lane) {
    for (int j0 = 16 * warp; j0 < 16 * warp + 16; j0 += 8) {
        float acc[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.0f;
        int tc[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) tc[c] = min(lane + 32 * c, n - 1);
#pragma unroll 4
        for (int r = 0; r < R; ++r) {
            const float4 lo = *reinterpret_cast<const float4*>(dz + r * GS + j0);
            const float4 hi = *reinterpret_cast<const float4*>(dz + r * GS + j0 + 4);
            const float d[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float v = x[r * xs + tc[c]];
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[i][c] = fmaf(d[i], v, acc[i][c]);
            }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int c = 0; c < 4; ++c)
                if (lane + 32 * c < n) G[(size_t)(j0 + i) * n + lane + 32 * c] = acc[i][c];
    }
}

static size_t grad_smem(int F) {
    return (size_t)((R + MLP_H) * grad_stride(F) + MLP_H * GS + 3 * R * GS + 2 * R) * 4;
}

__global__ void __launch_bounds__(GT) k_grad_partial(const float* __restrict__ P, int F, const float* __restrict__ feat,
                                                     const float* __restrict__ y, int m, float quantile,
                                                     float* __restrict__ partial) {
    extern __shared__ __align__(16) float sm[];
    const int FS = grad_stride(F);
    float* f_s = sm;                  // [R][FS]
    float* w1_s = f_s + R * FS;       // [H][FS]
    float* w2_s = w1_s + MLP_H * FS;  // [H][GS]
    float* h1_s = w2_s + MLP_H * GS;  // [R][GS]
    float* h2_s = h1_s + R * GS;      // [R][GS], then dz1
    float* dz2_s = h2_s + R * GS;     // [R][GS]
    float* out_s = dz2_s + R * GS;    // [R]
    float* g_s = out_s + R;           // [R] dL/dout
    float* dz1_s = h2_s;
    const Off o = offsets(F);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int r0 = blockIdx.x * R, rw = 4 * warp;
    for (int r = warp; r < R; r += GT / 32)
        for (int t = lane; t < F; t += 32) {
            if (r0 + r < m) cp4(f_s + r * FS + t, feat + (size_t)(r0 + r) * F + t);
            else f_s[r * FS + t] = 0.0f;
        }
    for (int u = warp; u < MLP_H; u += GT / 32)
        for (int t = lane; t < F; t += 32) cp4(w1_s + u * FS + t, P + o.w1 + (size_t)u * F + t);
    asm volatile("cp.async.commit_group;");
    for (int e = tid; e < MLP_H * MLP_H / 4; e += GT)
        cp16(w2_s + (e >> 5) * GS + 4 * (e & 31), P + o.w2 + 4 * (size_t)e);
    asm volatile("cp.async.commit_group;");
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    auto layer = [&](const float* x, int xs, const float* w, int ws, int n, const float* bias, float* out) {
        float acc[4][4];
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[0][c] = acc[1][c] = acc[2][c] = acc[3][c] = bias[lane + 32 * c];
        layer_tile(acc, x + rw * xs, xs, w + lane * ws, ws, n);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int c = 0; c < 4; ++c) out[(rw + i) * GS + lane + 32 * c] = fmaxf(acc[i][c], 0.0f);
    };
    layer(f_s, FS, w1_s, FS, F, P + o.b1, h1_s);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    layer(h1_s, GS, w2_s, GS, MLP_H, P + o.b2, h2_s);
    __syncthreads();
    if (tid < R) {
        float z = P[o.b3];
#pragma unroll 8
        for (int t = 0; t < MLP_H; t += 4) {
            const float4 h = *reinterpret_cast<const float4*>(h2_s + tid * GS + t);
            z = fmaf(P[o.w3 + t], h.x, z);
            z = fmaf(P[o.w3 + t + 1], h.y, z);
            z = fmaf(P[o.w3 + t + 2], h.z, z);
            z = fmaf(P[o.w3 + t + 3], h.w, z);
        }
        const int i = r0 + tid;
        // pinball loss ρ(y − out): d/dout = (1 − α) when out > y, −α otherwise
        g_s[tid] = i < m ? (z > y[i] ? 1.0f - quantile : -quantile) / (float)m : 0.0f;
    }
    __syncthreads();
    float* G = partial + (size_t)blockIdx.x * mlp_param_count(F);
    {
        const int j = tid & (MLP_H - 1);
        const float w3j = P[o.w3 + j];
        for (int r = tid / MLP_H; r < R; r += GT / MLP_H)
            dz2_s[r * GS + j] = h2_s[r * GS + j] > 0.0f ? g_s[r] * w3j : 0.0f;
        if (tid < MLP_H) {
            float gw3 = 0.0f;
            for (int r = 0; r < R; ++r) gw3 = fmaf(g_s[r], h2_s[r * GS + j], gw3);
            G[o.w3 + j] = gw3;
        } else if (tid == MLP_H) {
            float gb3 = 0.0f;
            for (int r = 0; r < R; ++r) gb3 += g_s[r];
            G[o.b3] = gb3;
        }
    }
    __syncthreads();
    // layer 2: dW2[j][t] = Σ_r dz2[r][j] h1[r][t], db2[j] = Σ_r dz2[r][j]
    weight_grad(G + o.w2, dz2_s, h1_s, GS, MLP_H, warp, lane);
    if (tid < MLP_H) {
        float gb = 0.0f;
        for (int r = 0; r < R; ++r) gb += dz2_s[r * GS + tid];
        G[o.b2 + tid] = gb;
    }
    {
        // dh1[r][j] = Σ_u dz2[r][u] W2[u][j], masked by the ReLU of layer 1
        float acc[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.0f;
#pragma unroll 2
        for (int u = 0; u < MLP_H; u += 4) {
            float4 a[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(dz2_s + (rw + i) * GS + u);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                float b[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) b[c] = w2_s[(u + q) * GS + lane + 32 * c];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float d = q == 0 ? a[i].x : q == 1 ? a[i].y : q == 2 ? a[i].z : a[i].w;
#pragma unroll
                    for (int c = 0; c < 4; ++c) acc[i][c] = fmaf(d, b[c], acc[i][c]);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int e = (rw + i) * GS + lane + 32 * c;
                dz1_s[e] = h1_s[e] > 0.0f ? acc[i][c] : 0.0f;  // (h2 is no longer read)
            }
    }
    __syncthreads();
    weight_grad(G + o.w1, dz1_s, f_s, FS, F, warp, lane);
    if (tid < MLP_H) {
        float gb = 0.0f;
        for (int r = 0; r < R; ++r) gb += dz1_s[r * GS + tid];
        G[o.b1 + tid] = gb;
    }
}

// The groups' gradients of one parameter, summed in group order (16 loads in flight).
__device__ __forceinline__ float sum_groups(const float* __restrict__ partial, int groups, size_t np, size_t p) {
    float s = 0.0f;
#pragma unroll 16
    for (int g = 0; g < groups; ++g) s += partial[(size_t)g * np + p];
    return s;
}

__global__ void k_grad_reduce(const float* __restrict__ partial, int groups, size_t np, float* __restrict__ grad) {
    const size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (p < np) grad[p] = sum_groups(partial, groups, np, p);
}

// The gradient sum and the Adam step it feeds, in one launch: a parameter's update needs nothing but
// its own sum, so the sum does not go through memory.
__global__ void k_adam(const float* __restrict__ partial, int groups, float* __restrict__ P, float* __restrict__ m1,
                       float* __restrict__ m2, size_t np, float lr, float bc1, float bc2) {
    const size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (p >= np) return;
    const float gp = sum_groups(partial, groups, np, p);
    const float a = 0.9f * m1[p] + 0.1f * gp;
    const float b = 0.999f * m2[p] + 0.001f * gp * gp;
    m1[p] = a;
    m2[p] = b;
    P[p] -= lr * (a / bc1) / (sqrtf(b / bc2) + 1e-8f);
}

__global__ void k_round_bf16(const float* __restrict__ P, float* __restrict__ Q, size_t np) {
    for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < np; p += (size_t)gridDim.x * blockDim.x)
        Q[p] = __bfloat162float(__float2bfloat16_rn(P[p]));
}

__global__ void k_block_min(const float* __restrict__ pred, const uint32_t* __restrict__ perm, int n,
                            float* __restrict__ tq) {
    const int Q = blockIdx.x;
    __shared__ float red[prune::QB];
    const int w = Q * prune::QB + threadIdx.x;
    red[threadIdx.x] = w < n ? pred[perm[w]] : CUDART_INF_F;
    __syncthreads();
    for (int s = prune::QB / 2; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s) red[threadIdx.x] = fminf(red[threadIdx.x], red[threadIdx.x + s]);
        __syncthreads();
    }
    if (threadIdx.x == 0) tq[Q] = red[0];
}

// ---- launchers ----------------------------------------------------------------------------------

cudaError_t features(const float* xsT, int np, int d, const float* centroids, int K, const uint32_t* rows, int m,
                     float* feat, cudaStream_t st) {
    if (m == 0) return cudaSuccess;
    if (K > FEAT_C) return cudaErrorInvalidValue;
    const size_t smem = (size_t)d * FEAT_C * 4;
    cudaError_t e = cudaFuncSetAttribute(k_features, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int dev = 0, sms = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    const int blocks = (m + 7) / 8 < 4 * sms ? (m + 7) / 8 : 4 * sms;
    k_features<<<blocks, 256, smem, st>>>(xsT, np, d, centroids, K, rows, m, feat); note_launch();
    return cudaGetLastError();
}

static size_t infer_smem(int F) {
    (void)F;
    return ((size_t)MLP_H * IKP + (size_t)MLP_H * IHP + (size_t)IR * IKP) * 2 + 3 * MLP_H * 4;
}

cudaError_t forward(const float* params, int F, const float* feat, int m, float* out, cudaStream_t st) {
    if (m == 0) return cudaSuccess;
    const size_t smem = infer_smem(F);
    cudaError_t e = cudaFuncSetAttribute(k_infer, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int dev = 0, sms = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    const int tiles = (m + IR - 1) / IR;
    k_infer<<<tiles < 2 * sms ? tiles : 2 * sms, IT, smem, st>>>(params, F, feat, m, out); note_launch();
    return cudaGetLastError();
}

static cudaError_t launch_partial(const float* params, int F, const float* feat, const float* y, int m, float quantile,
                                  float* partial, cudaStream_t st) {
    const size_t smem = grad_smem(F);
    cudaError_t e = cudaFuncSetAttribute(k_grad_partial, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k_grad_partial<<<(m + R - 1) / R, GT, smem, st>>>(params, F, feat, y, m, quantile, partial); note_launch();
    return cudaGetLastError();
}

cudaError_t gradient(const float* params, int F, const float* feat, const float* y, int m, float quantile,
                     float* partial, float* grad, cudaStream_t st) {
    cudaError_t e = launch_partial(params, F, feat, y, m, quantile, partial, st);
    if (e != cudaSuccess) return e;
    const size_t np = mlp_param_count(F);
    k_grad_reduce<<<(unsigned)((np + 127) / 128), 128, 0, st>>>(partial, (m + R - 1) / R, np, grad); note_launch();
    return cudaGetLastError();
}

cudaError_t train_step(float* params, int F, const float* feat, const float* y, int m, float quantile, float* partial,
                       float* m1, float* m2, float lr, int t, cudaStream_t st) {
    cudaError_t e = launch_partial(params, F, feat, y, m, quantile, partial, st);
    if (e != cudaSuccess) return e;
    const float bc1 = 1.0f - powf(0.9f, (float)t), bc2 = 1.0f - powf(0.999f, (float)t);
    const size_t np = mlp_param_count(F);
    k_adam<<<(unsigned)((np + 127) / 128), 128, 0, st>>>(partial, (m + R - 1) / R, params, m1, m2, np, lr, bc1, bc2); note_launch();
    return cudaGetLastError();
}

cudaError_t round_bf16(const float* params, float* params_bf, size_t np, cudaStream_t st) {
    k_round_bf16<<<64, 256, 0, st>>>(params, params_bf, np); note_launch();
    return cudaGetLastError();
}

cudaError_t block_min(const float* pred_orig, const uint32_t* perm, int n, float* tq, cudaStream_t st) {
    k_block_min<<<(n + prune::QB - 1) / prune::QB, prune::QB, 0, st>>>(pred_orig, perm, n, tq); note_launch();
    return cudaGetLastError();
}

}  // namespace mlp
}  // namespace costal
