// Locality order and block pruning: the column lists of the tensor-core and FP32 coarse passes, and the norm
// order of Tanimoto selection.
//
// The reference visits column blocks in index order and prunes only for Tanimoto selection, by norm
// windows (crates/costal-core/src/knn.rs:603-644, :272-283). This file gives the cosine path the same
// two levers, with bounds that hold for the exact scores:
//
//   cells     spherical k-means (K = 256 centroids, a seeded sample of rows, a few Lloyd steps with
//             deterministic centroid sums) and the cell of every row;
//   order     a working order: rows stably sorted by cell (ties by original index). The tensor
//             operands (or the FP32 pass's rows) are laid out in this order; candidates are mapped back to original indices.
//   geometry  for every 128-row query block Q and every column block B (128 working rows, or 256 for
//             lists longer than the sort takes; prune.h col_block) a
//             unit centre c and an angular radius r = max angle(row, c), in f64;
//   bound     for q ∈ Q, x ∈ B: angle(q, x) ≥ angle(c_Q, c_B) − r_Q − r_B (the angle is a metric on
//             the sphere), so cos(q, x) ≤ UB(Q, B) = cos(max(0, angle(c_Q, c_B) − r_Q − r_B − ξ)),
//             with ξ = 1e-6 rad covering the f32 rounding of the normalised rows (≤ 1e-7 rad); UB is
//             evaluated in f32 with directed roundings and margins for the f32 dot, acosf and cosf
//             (block_ub_f32), so it stays an upper bound;
//   row bound with M[Q][B] = the largest coarse score q·c_B over the rows q ∈ Q (tensor cores,
//             knn_tc.cu) and its margin δ: angle(q, c_B) ≥ acos(M + δ) for every q ∈ Q, so
//             cos(q, x) ≤ cos(max(0, acos(M + δ) − r_B − ξ)), evaluated like UB (row_ub_f32). It
//             drops the query block's radius, which the triangle inequality charges in full
//             although in d dimensions the rows spread mostly across the direction to c_B; the
//             lists use the smaller of the two bounds;
//   lists     for every Q, the column blocks with UB ≥ t_Q, sorted by UB descending (the closest
//             blocks first, so a query's threshold rises to its final value within the first tiles),
//             and ub_skip[Q] = the largest UB of a skipped block. A query is certified only if its
//             k-th exact score is strictly above ub_skip of its block; otherwise it is rescanned.

#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "fp32_tile.cuh"
#include "kernels.h"
#include "prune.h"

namespace costal {
namespace prune {

// ---- k-means ----------------------------------------------------------------------------------

// The sample (row j of it: row ⌊j·n/m⌋), row-major [m][d] and transposed [dp][mp] (zero padded), and the
// initial centroids: K evenly spaced sample rows, row-major and transposed [dp][K].
__global__ void k_sample(const float* __restrict__ xsR, int n, int d, int dp, int m, int mp, int K, float* __restrict__ rows,
                         float* __restrict__ rowsT, float* __restrict__ cent, float* __restrict__ centT) {
    auto source = [&](int j) { return (size_t)(((unsigned long long)j * (unsigned long long)n) / (unsigned long long)m); };
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < mp * dp; e += gridDim.x * blockDim.x) {
        const int t = e / mp, j = e - t * mp;  // (transposed: lanes run over the rows)
        const float v = j < m && t < d ? xsR[source(j) * d + t] : 0.0f;
        rowsT[e] = v;
        if (j < m && t < d) rows[(size_t)j * d + t] = v;
    }
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < K * dp; e += gridDim.x * blockDim.x) {
        const int t = e / K, c = e - t * K;
        const float v = t < d ? xsR[source((int)(((long long)c * m) / K)) * d + t] : 0.0f;
        centT[e] = v;
        if (t < d) cent[(size_t)c * d + t] = v;
    }
}

// Best centroid (largest dot with the unit centroid, ties to the smallest index) of every column of
// rowsT [dp][mp]: 128 rows per CTA against the 256 centroids (centT [dp][256]) on the 16 × 8 register
// tile, in two halves of 128 centroids. Every dot is one FMA chain in dimension order. One row per
// thread against broadcast centroids took a 16-byte shared load for every 4 FMAs: 1.83 ms at
// 2,000,000 × 40, 100 us for a 65,536-row sample; this tile 1 per 8 paired FMAs.
constexpr int KM_ROWS = 128;
__global__ void __launch_bounds__(128, 2) k_assign(const float* __restrict__ rowsT, int mp, int m, int dp,
                                                   const float* __restrict__ centT, uint32_t* __restrict__ assign) {
    using namespace fp32;
    static_assert(K_CENTROIDS == 256, "two halves of 128 centroids");
    extern __shared__ float4 km_s[];
    float* rows_s = reinterpret_cast<float*>(km_s);  // [dp][128]
    float* cent_s = rows_s + dp * KM_ROWS;           // [2][dp][128]
    const int r0 = blockIdx.x * KM_ROWS, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int e = threadIdx.x; e < dp * 32; e += 128)
        cp_async16(rows_s + e * 4, rowsT + (size_t)(e >> 5) * mp + r0 + (e & 31) * 4);
    for (int e = threadIdx.x; e < dp * 64; e += 128) {
        const int t = e >> 6, c4 = e & 63;
        cp_async16(cent_s + ((c4 >> 5) * dp + t) * 128 + (c4 & 31) * 4, centT + (size_t)t * 256 + c4 * 4);
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    const int tx = lane & 15, ty = 2 * warp + (lane >> 4);
    float best[16];
    int arg[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        best[i] = -CUDART_INF_F;
        arg[i] = 0;
    }
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
        unsigned long long acc[8][8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[i][j] = 0ull;
#pragma unroll 1
        for (int t = 0; t < dp; t += 8)
            fma8(reinterpret_cast<const ulonglong2*>(rows_s) + t * 32,
                 reinterpret_cast<const float4*>(cent_s + h * dp * 128) + t * 32, tx, ty, acc);
#pragma unroll
        for (int i = 0; i < 16; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) {  // ascending centroid indices
                const float v = tile_score(acc, i, j);
                if (v > best[i]) {
                    best[i] = v;
                    arg[i] = h * 128 + tile_col(j, tx);
                }
            }
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) {
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
            const float ob = __shfl_xor_sync(COSTAL_FULL_MASK, best[i], o);
            const int oa = __shfl_xor_sync(COSTAL_FULL_MASK, arg[i], o);
            const bool take = ob > best[i] || (ob == best[i] && oa < arg[i]);
            best[i] = take ? ob : best[i];
            arg[i] = take ? oa : arg[i];
        }
        const int r = r0 + tile_row(i, ty);
        if (tx == i && r < m) assign[r] = (uint32_t)arg[i];
    }
}

// One CTA per centroid: the normalised sum of its rows, summed in a fixed order (deterministic): the
// rows fall into 128 classes by (row / 4) mod 128, each class adds its rows in row order, and the 128
// class sums are combined by a fixed pairwise tree. Warp w takes classes 4w … 4w+3 one after the
// other (the adds wait for their rows: 32 warps a centroid hide that, 8 did not; the four classes side by
// side were slower, 24 against 19 us at 20,000 rows), lane t holding dimensions t and t + 32: the class's
// assignment words are loaded four per lane at once and its matches found by ballots, so the warp's
// branches are uniform and a row is read coalesced. An empty cluster keeps its previous centroid.
constexpr int UPD_T = 1024;
constexpr int UPD_CLASSES = 128;
constexpr int UPD_GROUPS = 128;  // word groups of a class: m ≤ 4 · 128 · 128 rows
static_assert(4 * UPD_CLASSES * UPD_GROUPS >= SAMPLE, "the centroid update covers the k-means sample");
__global__ void __launch_bounds__(UPD_T) k_centroid_update(const float* __restrict__ rows, int m, int d,
                                                           const uint32_t* __restrict__ assign, float* __restrict__ cent,
                                                           float* __restrict__ centT) {
    constexpr int NW = UPD_T / 32, CPW = UPD_CLASSES / NW;
    __shared__ float part[UPD_CLASSES][65];
    __shared__ int cnt_s[UPD_CLASSES];
    __shared__ float nrm;
    const int c = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m4 = m & ~3;
    for (int k = 0; k < CPW; ++k) {
        const int cls = warp * CPW + k;
        float s0 = 0.0f, s1 = 0.0f;
        int cnt = 0;
        auto add_row = [&](int i) {
            ++cnt;
            if (lane < d) s0 += rows[(size_t)i * d + lane];
            if (lane + 32 < d) s1 += rows[(size_t)i * d + lane + 32];
        };
        // the class's word groups q = 0 … 127 (rows 4·cls + 512·q …+3), four per lane, all loaded at
        // once; then the matches are added in row order: group by group (ballot, lowest lane first)
        // and within a group by row
        uint32_t mask[UPD_GROUPS / 32];
#pragma unroll
        for (int r = 0; r < UPD_GROUPS / 32; ++r) {
            const int i4 = 4 * cls + 4 * UPD_CLASSES * (r * 32 + lane);
            mask[r] = 0u;
            if (i4 < m4) {
                const uint4 a = *reinterpret_cast<const uint4*>(assign + i4);  // (the array is 256-byte aligned)
                mask[r] = (a.x == (uint32_t)c ? 1u : 0u) | (a.y == (uint32_t)c ? 2u : 0u) |
                          (a.z == (uint32_t)c ? 4u : 0u) | (a.w == (uint32_t)c ? 8u : 0u);
            }
        }
#pragma unroll
        for (int r = 0; r < UPD_GROUPS / 32; ++r) {
            unsigned any = __ballot_sync(COSTAL_FULL_MASK, mask[r] != 0u);
            while (any) {
                const int L = __ffs(any) - 1;
                any &= any - 1;
                unsigned mk = __shfl_sync(COSTAL_FULL_MASK, mask[r], L);
                const int i4 = 4 * cls + 4 * UPD_CLASSES * (r * 32 + L);
                while (mk) {
                    add_row(i4 + __ffs(mk) - 1);
                    mk &= mk - 1;
                }
            }
        }
        if (m4 + cls < m && assign[m4 + cls] == (uint32_t)c) add_row(m4 + cls);  // the last m mod 4 rows
        if (lane < d) part[cls][lane] = s0;
        if (lane + 32 < d) part[cls][lane + 32] = s1;
        if (lane == 0) cnt_s[cls] = cnt;
    }
    __syncthreads();
    for (int s = UPD_CLASSES / 2; s > 0; s >>= 1) {
        for (int e = threadIdx.x; e < s * d; e += UPD_T) {
            const int cls = e / d, t = e - cls * d;
            part[cls][t] += part[cls + s][t];
        }
        if ((int)threadIdx.x < s) cnt_s[threadIdx.x] += cnt_s[threadIdx.x + s];
        __syncthreads();
    }
    if (cnt_s[0] == 0) return;
    if (threadIdx.x == 0) {
        double nn = 0.0;
        for (int t = 0; t < d; ++t) nn += (double)part[0][t] * part[0][t];
        nrm = (float)sqrt(nn);
    }
    __syncthreads();
    if ((int)threadIdx.x < d && nrm > 0.0f) {
        const float v = part[0][threadIdx.x] / nrm;
        cent[(size_t)c * d + threadIdx.x] = v;
        centT[(size_t)threadIdx.x * K_CENTROIDS + c] = v;
    }
}

// ---- working order: stable counting sort of rows by cell -------------------------------------

// Chunks of 1,024 rows, one warp each: a histogram per chunk (hist [K][chunks]), every cell's counts
// scanned over the chunks, and the scatter: within a chunk a row's rank among the equal cells before it
// comes from a warp match. (One thread per chunk, walking its rows, took 0.5–0.8 ms at any n.)
constexpr int CHUNK = 1024;
constexpr int SORT_WARPS = 4;

__global__ void __launch_bounds__(32 * SORT_WARPS) k_cell_hist(const uint32_t* __restrict__ cell, int n, int K, int nch,
                                                               uint32_t* __restrict__ hist) {
    extern __shared__ uint32_t sort_s[];  // [SORT_WARPS][K]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, ch = blockIdx.x * SORT_WARPS + warp;
    uint32_t* h = sort_s + warp * K;
    for (int c = lane; c < K; c += 32) h[c] = 0u;
    __syncwarp();
    if (ch >= nch) return;
    const int end = min(n, (ch + 1) * CHUNK);
    for (int i = ch * CHUNK + lane; i < end; i += 32) atomicAdd(&h[cell[i]], 1u);
    __syncwarp();
    for (int c = lane; c < K; c += 32) hist[(size_t)c * nch + ch] = h[c];
}

// One CTA per cell: its chunk counts become exclusive offsets within the cell; total[c] = its rows.
__global__ void __launch_bounds__(256) k_cell_scan(uint32_t* __restrict__ hist, int nch, uint32_t* __restrict__ total) {
    __shared__ uint32_t wsum[8];
    uint32_t* row = hist + (size_t)blockIdx.x * nch;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t carry = 0;
    for (int b = 0; b < nch; b += 256) {
        const int e = b + threadIdx.x;
        const uint32_t v = e < nch ? row[e] : 0u;
        uint32_t x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(COSTAL_FULL_MASK, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) wsum[warp] = x;
        __syncthreads();
        uint32_t before = carry, all = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) {
            before += w < warp ? wsum[w] : 0u;
            all += wsum[w];
        }
        if (e < nch) row[e] = before + x - v;
        carry += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) total[blockIdx.x] = carry;
}

__global__ void __launch_bounds__(32 * SORT_WARPS) k_cell_scatter(const uint32_t* __restrict__ cell, int n, int K, int nch,
                                                                  const uint32_t* __restrict__ hist,
                                                                  const uint32_t* __restrict__ total,
                                                                  uint32_t* __restrict__ perm) {
    extern __shared__ uint32_t sort_s[];  // [K] cell starts, then [SORT_WARPS][K] the chunks' next positions
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, ch = blockIdx.x * SORT_WARPS + warp;
    uint32_t* start = sort_s;
    if (warp == 0) {  // exclusive scan of the cells' totals
        uint32_t carry = 0;
        for (int b = 0; b < K; b += 32) {
            const uint32_t v = b + lane < K ? total[b + lane] : 0u;
            uint32_t x = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(COSTAL_FULL_MASK, x, o);
                if (lane >= o) x += y;
            }
            if (b + lane < K) start[b + lane] = carry + x - v;
            carry += __shfl_sync(COSTAL_FULL_MASK, x, 31);
        }
    }
    __syncthreads();
    if (ch >= nch) return;
    uint32_t* next = sort_s + (1 + warp) * K;
    for (int c = lane; c < K; c += 32) next[c] = start[c] + hist[(size_t)c * nch + ch];
    __syncwarp();
    const int end = min(n, (ch + 1) * CHUNK);
    constexpr int AHEAD = 8;  // cells loaded at once: the ranks are a serial chain, their loads need not be
    uint32_t ahead[AHEAD];
    for (int i0 = ch * CHUNK; i0 < end; i0 += 32) {
        const int step = ((i0 - ch * CHUNK) >> 5) & (AHEAD - 1);
        if (step == 0) {
#pragma unroll
            for (int a = 0; a < AHEAD; ++a) ahead[a] = i0 + 32 * a + lane < end ? cell[i0 + 32 * a + lane] : 0xffffffffu;
        }
        const int i = i0 + lane;
        const bool live = i < end;
        uint32_t c = ahead[0];
#pragma unroll
        for (int a = 1; a < AHEAD; ++a) c = step == a ? ahead[a] : c;
        const unsigned peers = __match_any_sync(COSTAL_FULL_MASK, c);
        uint32_t base = 0;
        if (live) base = next[c];
        __syncwarp();
        if (live) {
            perm[base + __popc(peers & ((1u << lane) - 1u))] = (uint32_t)i;
            if (lane == __ffs(peers) - 1) next[c] = base + __popc(peers);
        }
        __syncwarp();
    }
}

// The stable order of n rows by cell (K cells). hist: K·⌈n/CHUNK⌉ words, total: K.
static cudaError_t sort_by_cell(const uint32_t* cell, int n, int K, uint32_t* hist, uint32_t* total, uint32_t* perm,
                                cudaStream_t st) {
    const int nch = (n + CHUNK - 1) / CHUNK, blocks = (nch + SORT_WARPS - 1) / SORT_WARPS;
    k_cell_hist<<<blocks, 32 * SORT_WARPS, (size_t)SORT_WARPS * K * 4, st>>>(cell, n, K, nch, hist); note_launch();
    k_cell_scan<<<K, 256, 0, st>>>(hist, nch, total); note_launch();
    k_cell_scatter<<<blocks, 32 * SORT_WARPS, (size_t)(SORT_WARPS + 1) * K * 4, st>>>(cell, n, K, nch, hist, total, perm);
    note_launch();
    return cudaGetLastError();
}

// The rows in working order, row-major: wrows[w] = xsR[perm[w]], whole rows at a time.
__global__ void k_gather_rows(const float* __restrict__ xsR, int d, const uint32_t* __restrict__ perm, int n,
                              float* __restrict__ wrows) {
    const size_t total = (size_t)n * d;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
        const size_t w = e / d;
        wrows[e] = xsR[(size_t)perm[w] * d + (e - w * d)];
    }
}

// ---- block geometry -------------------------------------------------------------------------------

// One CTA per block of `bs` consecutive working rows (wrows: the normalised rows in working order,
// row-major [n][d]; staged through shared memory): centre = normalised f64 sum (row order), radius = the
// largest angle between a row and the centre (f64). Rows past n are ignored. With center_f, the centre
// and radius go out in f32 too (transposed, and rounded up).
__global__ void __launch_bounds__(128) k_block_geom(const float* __restrict__ wrows, int d, int n, int bs,
                                                    double* __restrict__ center, double* __restrict__ radius,
                                                    float* __restrict__ center_f, float* __restrict__ radius_f) {
    extern __shared__ float rows_s[];  // [bs][d | 1]: an odd stride, so a warp's rows fall in 32 banks
    __shared__ double c_s[64];
    __shared__ double inv_s;
    __shared__ float cf_s[64];
    __shared__ float red[4];
    const int b = blockIdx.x, ds = d | 1;
    const int r0 = b * bs, nr = min(n, r0 + bs) - r0;
    for (int e = threadIdx.x; e < nr * d; e += 128) rows_s[(e / d) * ds + e % d] = wrows[(size_t)r0 * d + e];
    __syncthreads();
    if ((int)threadIdx.x < d) {
        double s = 0.0;
        for (int w = 0; w < nr; ++w) s += f64_of(rows_s[w * ds + threadIdx.x]);
        c_s[threadIdx.x] = s;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double nn = 0.0;
        for (int t = 0; t < d; ++t) nn += c_s[t] * c_s[t];
        inv_s = nn > 0.0 ? 1.0 / sqrt(nn) : 0.0;
    }
    __syncthreads();
    if ((int)threadIdx.x < d) {
        const double c = c_s[threadIdx.x] * inv_s;
        center[(size_t)b * d + threadIdx.x] = c;
        cf_s[threadIdx.x] = (float)c;
        if (center_f) center_f[(size_t)threadIdx.x * gridDim.x + b] = (float)c;  // [d][blocks]
    }
    __syncthreads();
    // The radius in f32 with a rigorous margin: the rows are unit vectors to within (d + 2)·2⁻²⁴, the
    // f32 centre is the f64 one to 2⁻²⁴ per component, and the f32 dot and norm accumulate at most
    // d·2⁻²⁴ of relative error each, so the f32 cosine is within (2d + 8)·2⁻²⁴ of the exact one; twice
    // that is subtracted before acosf (itself within a few ulp, covered by 1e-6 rad), and every step
    // rounds up. A zero row has cosine 0 with everything: angle π/2 covers it.
    const float margin = (float)(2 * d + 8) * 0x1p-23f;
    float worst = 0.0f;
    for (int w = threadIdx.x; w < nr; w += 128) {
        const float* row = rows_s + w * ds;
        float dot = 0.0f, nn = 0.0f;
        for (int t = 0; t < d; ++t) {
            const float v = row[t];
            dot = fmaf(v, cf_s[t], dot);
            nn = fmaf(v, v, nn);
        }
        float ang = 1.57079637f;  // ≥ π/2
        if (nn > 0.0f) {
            const float cs = __fsub_rd(__fdiv_rd(dot, __fsqrt_ru(nn)), margin);
            ang = __fadd_ru(acosf(fminf(1.0f, fmaxf(-1.0f, cs))), 1e-6f);
        }
        worst = fmaxf(worst, ang);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) worst = fmaxf(worst, __shfl_xor_sync(COSTAL_FULL_MASK, worst, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = worst;
    __syncthreads();
    if (threadIdx.x == 0) {
        worst = fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3]));
        radius[b] = (double)worst;
        if (radius_f) radius_f[b] = worst;
    }
}

// ---- per-query-block lists ------------------------------------------------------------------------

constexpr int LIST_T = 512;
constexpr double XI = 1e-6;

// A list sort's shape: KPT keys per thread over LIST_T threads (16 → 8,192 column blocks, two CTAs
// per SM; 32 → 16,384, one CTA per SM with the keys in its registers). A key is 32 bits: a level of
// SBITS = 32 − ID_BITS bits above the complemented block id (ID_BITS bits). Levels [1, ONE) hold a
// bound u < 1 rounded up to a multiple of Q = 2 / ONE (u ≤ level·Q − 1 + Q); levels [ONE, 2·ONE) hold
// the blocks whose bound is 1, nearest centre first. Descending keys: larger bound first, then (at
// bound 1) smaller centre angle, then smaller block id.
template <int KPT>
struct ListShape {
    static constexpr int N = LIST_T * KPT;
    static constexpr int ID_BITS = KPT <= 16 ? 13 : 14;
    static constexpr uint32_t ID_MAX = (1u << ID_BITS) - 1u;
    static constexpr int SBITS = 32 - ID_BITS;
    static constexpr uint32_t ONE = 1u << (SBITS - 1);     // first level of the bound-1 range
    static constexpr float SCALE = (float)(1u << (SBITS - 2));  // levels per unit of (u + 1)
};

// The key of column block b with bound u (≤ 1) and centre angle φ (0 for a padding key never occurs:
// every key of a kept block is non-zero).
template <int KPT>
__device__ __forceinline__ uint32_t list_key(float u, float phi, int b) {
    using LS = ListShape<KPT>;
    uint32_t level;
    if (u >= 1.0f) {
        const float q = fmaxf(0.0f, phi) * ((float)LS::ONE / 3.14159265f);
        level = (2u * LS::ONE - 1u) - (uint32_t)fminf((float)(LS::ONE - 1u), q);
    } else {
        // ⌊(u + 1)·SCALE⌋ with u + 1 rounded up: level·Q − 1 + Q ≥ u holds for the level kept
        const float f = floorf(__fadd_ru(fmaxf(u, -1.0f), 1.0f) * LS::SCALE);
        level = (uint32_t)fminf((float)(LS::ONE - 1u), fmaxf(1.0f, f));
    }
    return (level << LS::ID_BITS) | (LS::ID_MAX - (uint32_t)b);
}

// The bound a key stands for: 1 in the bound-1 range, else the top of its level (exact in f32).
template <int KPT>
__device__ __forceinline__ float key_bound(uint32_t key) {
    using LS = ListShape<KPT>;
    const uint32_t level = key >> LS::ID_BITS;
    if (level >= LS::ONE) return 1.0f;
    return (float)(level + 1u) * (1.0f / LS::SCALE) - 1.0f;
}

// The bound in f32 for one (query block, column block) pair, rigorous for the f64 geometry: the
// f32 FMA dot of the two unit centres (each rounded to f32) is within (d + 2)·2⁻²⁴ of the f64 value,
// so acos(dot + δ) with δ = (d + 4)·2⁻²³, the sum rounded up, never exceeds the centres' angle;
// acosf and cosf are within a few ulp, covered by 1e-6 on each side; every subtraction rounds down
// and the final addition up. Radii arrive rounded up to f32.
// Also returns (in *phi_out) the centres' angle, used only to order blocks of equal bound.
__device__ __forceinline__ float block_ub_f32(const float* cq, float rq, const float* cb, int cstride, float rb, int d,
                                             float* phi_out = nullptr) {
    float dot = 0.0f;
    for (int t = 0; t < d; ++t) dot = fmaf(cq[t], cb[(size_t)t * cstride], dot);
    const float delta = (float)(d + 4) * 0x1p-23f;
    const float c = fminf(1.0f, __fadd_ru(dot, delta));
    const float phi = __fsub_rd(acosf(c), 1e-6f);
    if (phi_out) *phi_out = phi;
    const float th = __fsub_rd(__fsub_rd(__fsub_rd(phi, rq), rb), (float)XI);
    if (th <= 0.0f) return 1.0f;
    return fminf(1.0f, __fadd_ru(cosf(th), 1e-6f));
}

// The per-row bound in f32 from M = max over the query block's rows of the coarse q·c_B and its
// margin δ (M + δ ≥ the largest exact cosine of a row with c_B); radii arrive rounded up to f32,
// acosf and cosf are covered by 1e-6 on each side, subtractions round down, the last addition up.
__device__ __forceinline__ float row_ub_f32(float m, float delta, float rb) {
    const float c = fmaxf(-1.0f, fminf(1.0f, __fadd_ru(m, delta)));
    const float th = __fsub_rd(__fsub_rd(__fsub_rd(acosf(c), 1e-6f), rb), (float)XI);
    if (th <= 0.0f) return 1.0f;
    return fminf(1.0f, __fadd_ru(cosf(th), 1e-6f));
}

// Compare-exchange of list keys (descending) at a register distance S within a thread's run.
template <int S, int KPT>
__device__ __forceinline__ void cx_regs(uint32_t (&v)[KPT], int base, int size) {
#pragma unroll
    for (int j = 0; j < KPT; ++j) {
        const int p = j ^ S;
        if (p > j) {
            const bool desc = ((base + j) & size) == 0;
            const uint32_t a = v[j], b = v[p];
            const uint32_t hi = max(a, b), lo = min(a, b);
            v[j] = desc ? hi : lo;
            v[p] = desc ? lo : hi;
        }
    }
}

// Bitonic sort (descending) of the CTA's LIST_T·KPT keys, KPT per thread at positions base..base+KPT−1:
// compare-exchanges in registers, by warp shuffles, or through shared memory (xk) by distance.
template <int KPT>
__device__ __forceinline__ void block_sort_keys(uint32_t (&v)[KPT], uint32_t* xk, int base, int lane) {
    constexpr int N = LIST_T * KPT;
    for (int size = 2; size <= N; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            if (stride >= KPT * 32) {  // across warps
                __syncthreads();
#pragma unroll
                for (int j = 0; j < KPT; ++j) xk[base + j] = v[j];
                __syncthreads();
#pragma unroll
                for (int j = 0; j < KPT; ++j) {
                    const int e = base + j;
                    const uint32_t o = xk[e ^ stride];
                    const bool keep_max = ((e & stride) == 0) == ((e & size) == 0);
                    const uint32_t hi = max(v[j], o), lo = min(v[j], o);
                    v[j] = keep_max ? hi : lo;
                }
            } else if (stride >= KPT) {  // within the warp
                const int lstride = stride / KPT;
#pragma unroll
                for (int j = 0; j < KPT; ++j) {
                    const int e = base + j;
                    const uint32_t o = __shfl_xor_sync(COSTAL_FULL_MASK, v[j], lstride);
                    const bool keep_max = ((lane & lstride) == 0) == ((e & size) == 0);
                    const uint32_t hi = max(v[j], o), lo = min(v[j], o);
                    v[j] = keep_max ? hi : lo;
                }
            } else if (stride == 16) {
                if constexpr (KPT > 16) cx_regs<16>(v, base, size);
            } else if (stride == 8) {
                if constexpr (KPT > 8) cx_regs<8>(v, base, size);
            } else if (stride == 4) {
                if constexpr (KPT > 4) cx_regs<4>(v, base, size);
            } else if (stride == 2) {
                cx_regs<2>(v, base, size);
            } else {
                cx_regs<1>(v, base, size);
            }
        }
    }
}

// The sorted keys out (keys of ListShape<KPT_ALL>, KPT per thread): list position e holds block
// ID_MAX − (low ID_BITS bits) and the bound its level stands for.
template <int KPT, int KPT_ALL>
__device__ __forceinline__ void write_keys(const uint32_t (&v)[KPT], int base, unsigned nk, uint32_t* out, float* out_ub) {
    using LS = ListShape<KPT_ALL>;
#pragma unroll
    for (int j = 0; j < KPT; ++j) {
        const unsigned e = (unsigned)(base + j);
        if (e < nk) {
            out[e] = LS::ID_MAX - (v[j] & LS::ID_MAX);
            out_ub[e] = key_bound<KPT_ALL>(v[j]);
        }
    }
}

// Compact the kept keys (non-zero) of every thread into xk[0 .. kept) in any order, zero-fill up to
// LIST_T·KPT, and load KPT of them per thread.
template <int KPT, int KPT_ALL>
__device__ __forceinline__ void compact_keys(const uint32_t (&all)[KPT_ALL], uint32_t (&v)[KPT], uint32_t* xk,
                                             unsigned* slot, unsigned nk, int base) {
    constexpr int N = LIST_T * KPT;
    for (int e = threadIdx.x + (int)nk; e < N; e += LIST_T) xk[e] = 0u;
#pragma unroll
    for (int j = 0; j < KPT_ALL; ++j)
        if (all[j]) xk[atomicAdd(slot, 1u)] = all[j];
    __syncthreads();
#pragma unroll
    for (int j = 0; j < KPT; ++j) v[j] = xk[base + j];
    __syncthreads();  // every thread has its keys before the sort reuses xk
}

// One CTA per query block: the upper bound against every column block; the blocks kept (UB ≥ t_Q)
// sorted by (UB desc, centre angle asc at UB = 1, block asc) with their bounds rounded up to the keys'
// levels — a bitonic sort of 32-bit keys, 16 per thread, exchanged in registers, by warp shuffles or
// through shared memory by distance — and the largest UB of a skipped block. Lists longer than the
// shape's N stay in block order with bounds +inf.
template <int KPT_ALL, bool TANI>
__global__ void __launch_bounds__(LIST_T, KPT_ALL <= 16 ? 2 : 1)
    k_block_lists(const double* __restrict__ qcenter, const double* __restrict__ qradius,
                  const float* __restrict__ ccenter_f, const float* __restrict__ cradius_f, int nqb, int ncb, int d,
                  const float* __restrict__ tq, const float* __restrict__ rowmax, const float* __restrict__ rm_delta,
                  const float2* __restrict__ qnorm, const float2* __restrict__ cnorm, int use_cos,
                  uint32_t* __restrict__ lists, float* __restrict__ list_ub, uint32_t* __restrict__ counts,
                  uint32_t* __restrict__ weight, float* __restrict__ ub_skip,
                  unsigned long long* __restrict__ skipped_total) {
    using LS = ListShape<KPT_ALL>;
    extern __shared__ uint32_t xk[];  // [LS::N] exchange buffer
    __shared__ float cq[64];
    __shared__ unsigned kept, slot, near;
    __shared__ int skip_max_bits;
    const int Q = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
    if ((!TANI || use_cos) && tid < d) cq[tid] = (float)qcenter[(size_t)Q * d + tid];
    if (tid == 0) {
        kept = 0;
        slot = 0;
        near = 0;
        skip_max_bits = __float_as_int(-CUDART_INF_F);
    }
    __syncthreads();
    float rq = 0.0f;
    if (!TANI || use_cos) {
        rq = (float)qradius[Q];
        if ((double)rq < qradius[Q]) rq = nextafterf(rq, CUDART_INF_F);
    }
    const float2 nq = TANI ? qnorm[Q] : make_float2(0.0f, 0.0f);
    const float t = tq ? tq[Q] : -CUDART_INF_F;
    const float* rm = rowmax ? rowmax + (size_t)Q * ncb : nullptr;
    const float delta = rowmax ? *rm_delta : 0.0f;
    // the smaller of the cone bound and the per-row bound (without cosine bounds 1, all at one angle);
    // for Tanimoto selection the bound on T that it and the blocks' norms give
    auto bound = [&](int b, float* phi) {
        float u = 1.0f;
        if (!TANI || use_cos) {
            u = block_ub_f32(cq, rq, ccenter_f + b, ncb, cradius_f[b], d, phi);
            if (rm) u = fminf(u, row_ub_f32(rm[b], delta, cradius_f[b]));
        } else if (phi) {
            *phi = 0.0f;
        }
        return TANI ? tani_ub_f32(u, nq, cnorm[b]) : u;
    };
    uint32_t* out = lists + (size_t)Q * ncb;
    float* out_ub = list_ub + (size_t)Q * ncb;
    if (ncb > LS::N) {
        if (tid == 0) {
            unsigned c = 0;
            for (int b = 0; b < ncb; ++b) {
                const float u = bound(b, nullptr);
                if (u >= t) {
                    out_ub[c] = CUDART_INF_F;  // block order: the bounds do not decrease along the list
                    out[c++] = (uint32_t)b;
                } else {
                    skip_max_bits = max(skip_max_bits, __float_as_int(fmaxf(u, 0.0f)));
                }
            }
            kept = c;
        }
    } else {
        const int base = tid * KPT_ALL;
        uint32_t v[KPT_ALL];
        unsigned my_kept = 0, my_near = 0;
        int my_skip = __float_as_int(-CUDART_INF_F);
        // keys are computed for blocks j·LIST_T + tid (coalesced reads of the transposed centres); the
        // sort does not care where each key starts
#pragma unroll
        for (int j = 0; j < KPT_ALL; ++j) {
            const int b = j * LIST_T + tid;
            v[j] = 0u;  // absent or skipped: sorts last
            if (b < ncb) {
                float phi;
                const float u = bound(b, &phi);
                if (u >= t) {
                    ++my_kept;
                    my_near += u >= 0.9f ? 1u : 0u;
                    // ties of the bound at 1 (e.g. every block of the query's own cluster) go nearest
                    // centre first, then by block
                    v[j] = list_key<KPT_ALL>(u, phi, b);
                } else {
                    // a skipped block's bound, clamped at 0 so that the int order of the bits is the float order
                    my_skip = max(my_skip, __float_as_int(fmaxf(u, 0.0f)));
                }
            }
        }
        atomicAdd(&kept, my_kept);
        atomicAdd(&near, my_near);
        atomicMax(&skip_max_bits, my_skip);
        __syncthreads();  // kept is final
        const unsigned nk = kept;
        // Short lists (a learned threshold skips most blocks) sort only their kept keys, compacted.
        if (nk <= (unsigned)(LIST_T * 4)) {
            uint32_t w[4];
            compact_keys<4>(v, w, xk, &slot, nk, tid * 4);
            block_sort_keys<4>(w, xk, tid * 4, lane);
            write_keys<4, KPT_ALL>(w, tid * 4, nk, out, out_ub);
        } else if (nk <= (unsigned)(LIST_T * 8)) {
            uint32_t w[8];
            compact_keys<8>(v, w, xk, &slot, nk, tid * 8);
            block_sort_keys<8>(w, xk, tid * 8, lane);
            write_keys<8, KPT_ALL>(w, tid * 8, nk, out, out_ub);
        } else if (KPT_ALL > 16 && nk <= (unsigned)(LIST_T * 16)) {
            uint32_t w[16];
            compact_keys<16>(v, w, xk, &slot, nk, tid * 16);
            block_sort_keys<16>(w, xk, tid * 16, lane);
            write_keys<16, KPT_ALL>(w, tid * 16, nk, out, out_ub);
        } else {
            // the keys start interleaved over all N positions, so the sort covers all of them
            block_sort_keys<KPT_ALL>(v, xk, base, lane);
            write_keys<KPT_ALL, KPT_ALL>(v, base, nk, out, out_ub);
        }
    }
    __syncthreads();
    if (tid == 0) {
        counts[Q] = kept;
        weight[Q] = near;
        ub_skip[Q] = __int_as_float(skip_max_bits);
        if (skipped_total) atomicAdd(skipped_total, (unsigned long long)(ncb - (int)kept));
    }
}

// The query blocks by descending weight (the list entries with a bound of 0.9 or more, a guess at how far
// the block's list will be walked), in 1,024 classes: launched in this order the long lists start first and
// the short ones fill the last wave. One CTA; the order inside a class does not matter.
__global__ void __launch_bounds__(1024) k_block_order(const uint32_t* __restrict__ weight, int nqb, int ncb,
                                                      uint32_t* __restrict__ order) {
    __shared__ uint32_t next[1024], wsum[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    auto cls = [&](int Q) { return 1023 - (int)((unsigned long long)weight[Q] * 1023ull / (unsigned)max(ncb, 1)); };
    next[tid] = 0;
    __syncthreads();
    for (int Q = tid; Q < nqb; Q += 1024) atomicAdd(&next[cls(Q)], 1u);
    __syncthreads();
    const uint32_t v = next[tid];
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(COSTAL_FULL_MASK, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    uint32_t before = 0;
    for (int w = 0; w < warp; ++w) before += wsum[w];
    __syncthreads();
    next[tid] = before + x - v;
    __syncthreads();
    for (int Q = tid; Q < nqb; Q += 1024) order[atomicAdd(&next[cls(Q)], 1u)] = (uint32_t)Q;
}

// The per-row certificate floor from pruning: ub_skip of the row's query block, or −∞.
__global__ void k_row_ub(const uint32_t* __restrict__ perm, int n, const float* __restrict__ ub_skip,
                         double* __restrict__ row_ub) {
    const int w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= n) return;
    const float u = ub_skip[w / 128];
    row_ub[perm[w]] = u == -CUDART_INF_F ? -CUDART_INF : (double)u;
}

}  // namespace prune
}  // namespace costal

namespace costal {
namespace prune {

namespace {
inline size_t a256(size_t b) { return (b + 255) & ~(size_t)255; }
}  // namespace

bool supported(int d) { return d >= 1 && d <= 64; }

namespace {
struct Scratch {
    float *sample_rows, *sample_T, *centT;
    uint32_t *sample_assign, *hist, *total;
};

// The workspace's layout (base NULL: only its size).
size_t carve(void* base, int n, int d, Plan& P, Scratch& S) {
    const int K = K_CENTROIDS, cb = col_block(n), dp = coarse_dpad(d);
    const int m = n < SAMPLE ? n : SAMPLE, mp = (m + KM_ROWS - 1) / KM_ROWS * KM_ROWS;
    const size_t nqb = (size_t)(n + QB - 1) / QB, ncb = (size_t)(n + cb - 1) / cb, nch = (size_t)(n + CHUNK - 1) / CHUNK;
    size_t off = 0;
    auto take = [&](auto*& p, size_t count) {
        p = reinterpret_cast<std::remove_reference_t<decltype(p)>>(static_cast<char*>(base) + off);
        off += a256(count * sizeof(*p));
    };
    P.n = n;
    P.d = d;
    P.K = K;
    P.nqb = (int)nqb;
    P.ncb = (int)ncb;
    P.cb = cb;
    take(P.perm, n);
    take(P.cell, n);
    take(P.centroids, (size_t)K * d);
    take(P.ccenter, ncb * d);
    take(P.cradius, ncb);
    take(P.ccenter_f, ncb * d);
    take(P.cradius_f, ncb);
    if (cb == QB) {  // query and column blocks are the same rows
        P.qcenter = P.ccenter;
        P.qradius = P.cradius;
    } else {
        take(P.qcenter, nqb * d);
        take(P.qradius, nqb);
    }
    take(P.lists, nqb * ncb);
    take(P.list_ub, nqb * ncb);
    take(P.counts, nqb);
    take(P.weight, nqb);
    take(P.order, nqb);
    take(P.ub_skip, nqb);
    take(P.row_ub, n);
    take(P.tq, nqb);
    take(P.wrows, (size_t)n * d);
    take(S.sample_rows, (size_t)m * d);
    take(S.sample_T, (size_t)mp * dp);
    take(S.centT, (size_t)K * dp);
    take(S.sample_assign, m);
    take(S.hist, nch * K);
    take(S.total, K);
    return off;
}
}  // namespace

size_t workspace_bytes(int n, int d) {
    Plan P{};
    Scratch S{};
    return carve(nullptr, n, d, P, S);
}

cudaError_t build_order(void* ws, const float* xsT, const float* xsR, int n, int np, int d, cudaStream_t st, Plan& P) {
    const int K = K_CENTROIDS, dp = coarse_dpad(d);
    const int m = n < SAMPLE ? n : SAMPLE, mp = (m + KM_ROWS - 1) / KM_ROWS * KM_ROWS;
    Scratch S{};
    carve(ws, n, d, P, S);
    const size_t asm_ = (size_t)dp * (KM_ROWS + K) * 4;
    const size_t gsm = (size_t)P.cb * (d | 1) * 4;
    cudaError_t e;
    if ((e = cudaFuncSetAttribute(k_assign, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)asm_)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(k_block_geom, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gsm)) != cudaSuccess) return e;
    k_sample<<<std::min((mp * dp + 255) / 256, 4096), 256, 0, st>>>(xsR, n, d, dp, m, mp, K, S.sample_rows, S.sample_T,
                                                                    P.centroids, S.centT); note_launch();
    for (int it = 0; it < LLOYD_STEPS; ++it) {
        k_assign<<<mp / KM_ROWS, 128, asm_, st>>>(S.sample_T, mp, m, dp, S.centT, S.sample_assign); note_launch();
        k_centroid_update<<<K, UPD_T, 0, st>>>(S.sample_rows, m, d, S.sample_assign, P.centroids, S.centT); note_launch();
    }
    k_assign<<<np / KM_ROWS, 128, asm_, st>>>(xsT, np, n, dp, S.centT, P.cell); note_launch();
    if ((e = sort_by_cell(P.cell, n, K, S.hist, S.total, P.perm, st)) != cudaSuccess) return e;
    k_gather_rows<<<(unsigned)std::min<size_t>(((size_t)n * d + 255) / 256, 16 * 1024), 256, 0, st>>>(xsR, d, P.perm, n,
                                                                                                      P.wrows); note_launch();
    k_block_geom<<<P.ncb, 128, gsm, st>>>(P.wrows, d, n, P.cb, P.ccenter, P.cradius, P.ccenter_f, P.cradius_f); note_launch();
    if (P.cb != QB) {
        k_block_geom<<<P.nqb, 128, (size_t)QB * (d | 1) * 4, st>>>(P.wrows, d, n, QB, P.qcenter, P.qradius, nullptr, nullptr);
        note_launch();
    }
    return cudaGetLastError();
}

// The smallest and largest positive norm (order-preserving u64 bits of positive doubles).
__global__ void k_norm_range(const double* __restrict__ norms, int n, unsigned long long* __restrict__ range) {
    unsigned long long lo = ~0ull, hi = 0ull;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double a = norms[i];
        if (a > 0.0) {
            const unsigned long long b = (unsigned long long)__double_as_longlong(a);
            lo = min(lo, b);
            hi = max(hi, b);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = min(lo, __shfl_xor_sync(COSTAL_FULL_MASK, lo, o));
        hi = max(hi, __shfl_xor_sync(COSTAL_FULL_MASK, hi, o));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMin(&range[0], lo);
        atomicMax(&range[1], hi);
    }
}

// Bucket of every row: 0 for a zero row, else 1 + ⌊(NORM_BUCKETS − 2)·log(a/lo)/log(hi/lo)⌋.
__global__ void k_norm_bucket(const double* __restrict__ norms, int n, const unsigned long long* __restrict__ range,
                              uint32_t* __restrict__ cell) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double a = norms[i];
    const double lo = __longlong_as_double((long long)range[0]), hi = __longlong_as_double((long long)range[1]);
    uint32_t b = 0;
    if (a > 0.0) {
        const double span = hi > lo ? log(hi / lo) : 1.0;
        const double f = log(a / lo) / span * (double)(NORM_BUCKETS - 2);
        b = 1u + (uint32_t)fmin(fmax(f, 0.0), (double)(NORM_BUCKETS - 2));
    }
    cell[i] = b;
}

// The norm range of each block of `bs` working rows, rounded outward to f32 (one warp per block).
__global__ void k_block_norms(const double* __restrict__ norms, const uint32_t* __restrict__ perm, int n, int bs, int nb,
                              float2* __restrict__ range) {
    const int b = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (b >= nb) return;
    float lo = CUDART_INF_F, hi = 0.0f;
    for (int w = b * bs + lane; w < min(n, (b + 1) * bs); w += 32) {
        const double a = norms[perm[w]];
        lo = fminf(lo, __double2float_rd(a));
        hi = fmaxf(hi, __double2float_ru(a));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(COSTAL_FULL_MASK, lo, o));
        hi = fmaxf(hi, __shfl_xor_sync(COSTAL_FULL_MASK, hi, o));
    }
    if (lane == 0) range[b] = make_float2(lo, hi);
}

cudaError_t block_norms(const double* norms, Plan& P, float2* ranges, cudaStream_t st) {
    k_block_norms<<<(P.ncb + 7) / 8, 256, 0, st>>>(norms, P.perm, P.n, P.cb, P.ncb, ranges); note_launch();
    P.cnorm = P.qnorm = ranges;
    if (P.cb != QB) {
        k_block_norms<<<(P.nqb + 7) / 8, 256, 0, st>>>(norms, P.perm, P.n, QB, P.nqb, ranges + P.ncb); note_launch();
        P.qnorm = ranges + P.ncb;
    }
    return cudaGetLastError();
}

// Over a strided sample of up to 1,024 rows: share[0] = the pairs of live rows, share[1] = those whose
// norms' quotient lies inside the window of a Tanimoto score of 0.9 (ρ + 1/ρ ≤ 1.9 / 0.9).
__global__ void __launch_bounds__(1024) k_norm_window_share(const double* __restrict__ norms, int n, unsigned* __restrict__ share) {
    __shared__ float a_s[1024];
    const int m = min(n, 1024), i = threadIdx.x;
    a_s[i] = i < m ? (float)norms[(size_t)i * n / m] : 0.0f;
    __syncthreads();
    unsigned all = 0, in = 0;
    if (a_s[i] > 0.0f)
        for (int j = 0; j < m; ++j) {
            const float b = a_s[j], a = a_s[i];
            if (b > 0.0f) {
                ++all;
                in += a * a + b * b <= (1.9f / 0.9f) * a * b ? 1u : 0u;
            }
        }
    atomicAdd(&share[0], all);
    atomicAdd(&share[1], in);
}

cudaError_t norm_window_share(const double* norms, int n, unsigned* share, cudaStream_t st) {
    k_norm_window_share<<<1, 1024, 0, st>>>(norms, n, share); note_launch();
    return cudaGetLastError();
}

size_t norm_order_bytes(int n) {
    const size_t nch = (size_t)(n + CHUNK - 1) / CHUNK;
    return a256((size_t)n * 4) + a256(nch * NORM_BUCKETS * 4) + a256((NORM_BUCKETS + 1) * 4) + 256;
}

static cudaError_t norm_order(const double* norms, int n, void* ws, uint32_t* perm, cudaStream_t st) {
    char* p = static_cast<char*>(ws);
    const int nch = (n + CHUNK - 1) / CHUNK;
    uint32_t* cell = reinterpret_cast<uint32_t*>(p);
    p += a256((size_t)n * 4);
    uint32_t* hist = reinterpret_cast<uint32_t*>(p);
    p += a256((size_t)nch * NORM_BUCKETS * 4);
    uint32_t* start = reinterpret_cast<uint32_t*>(p);
    p += a256((NORM_BUCKETS + 1) * 4);
    unsigned long long* range = reinterpret_cast<unsigned long long*>(p);
    cudaError_t e = cudaMemsetAsync(range, 0xff, 8, st);  // smallest: all ones
    if (e == cudaSuccess) e = cudaMemsetAsync(range + 1, 0, 8, st);  // largest: zero
    if (e != cudaSuccess) return e;
    k_norm_range<<<std::min((n + 255) / 256, 1024), 256, 0, st>>>(norms, n, range); note_launch();
    k_norm_bucket<<<(n + 255) / 256, 256, 0, st>>>(norms, n, range, cell); note_launch();
    return sort_by_cell(cell, n, NORM_BUCKETS, hist, start, perm, st);
}

cudaError_t norm_plan(void* ws, const double* norms, int n, int d, void* norm_ws, cudaStream_t st, Plan& P) {
    Scratch S{};
    carve(ws, n, d, P, S);
    P.norm_only = true;
    return norm_order(norms, n, norm_ws, P.perm, st);
}

// ends[t] = (the smallest lower end of ranges[t …], the largest upper end of ranges[… t]). One CTA.
__global__ void __launch_bounds__(1024) k_walk_ends(const float2* __restrict__ ranges, int tiles, float2* __restrict__ ends) {
    __shared__ float lo_s[1024], hi_s[1024];
    const int tid = threadIdx.x, per = (tiles + 1023) / 1024;
    const long long a = min((long long)tid * per, (long long)tiles), b = min(a + per, (long long)tiles);
    float lo = CUDART_INF_F, hi = 0.0f;
    for (long long t = a; t < b; ++t) {
        lo = fminf(lo, ranges[t].x);
        hi = fmaxf(hi, ranges[t].y);
    }
    for (int o = 1; o < 1024; o <<= 1) {  // the threads' shares, scanned from both ends
        lo_s[tid] = lo;
        hi_s[tid] = hi;
        __syncthreads();
        if (tid + o < 1024) lo = fminf(lo, lo_s[tid + o]);
        if (tid >= o) hi = fmaxf(hi, hi_s[tid - o]);
        __syncthreads();
    }
    lo_s[tid] = lo;
    hi_s[tid] = hi;
    __syncthreads();
    lo = tid < 1023 ? lo_s[tid + 1] : CUDART_INF_F;
    hi = tid > 0 ? hi_s[tid - 1] : 0.0f;
    for (long long t = a; t < b; ++t) ends[t].y = hi = fmaxf(hi, ranges[t].y);
    for (long long t = b - 1; t >= a; --t) ends[t].x = lo = fminf(lo, ranges[t].x);
}

size_t norm_walk_bytes(int n) {
    const size_t tiles = ((size_t)n + QB - 1) / QB;
    return a256((size_t)n * 4) + 2 * a256(tiles * 8) + norm_order_bytes(n);
}

cudaError_t norm_walk(void* ws, const double* norms, int n, cudaStream_t st, Walk& W) {
    const int tiles = (n + QB - 1) / QB;
    char* p = static_cast<char*>(ws);
    uint32_t* perm = reinterpret_cast<uint32_t*>(p);
    p += a256((size_t)n * 4);
    float2* ranges = reinterpret_cast<float2*>(p);
    p += a256((size_t)tiles * 8);
    float2* ends = reinterpret_cast<float2*>(p);
    p += a256((size_t)tiles * 8);
    cudaError_t e = norm_order(norms, n, p, perm, st);
    if (e != cudaSuccess) return e;
    k_block_norms<<<(tiles + 7) / 8, 256, 0, st>>>(norms, perm, n, QB, tiles, ranges); note_launch();
    k_walk_ends<<<1, 1024, 0, st>>>(ranges, tiles, ends); note_launch();
    W.perm = perm;
    W.ranges = ranges;
    W.ends = ends;
    return cudaGetLastError();
}

static_assert(ListShape<16>::N == LIST_FAST && ListShape<32>::N == LIST_MAX, "the lists' limits are their sorts'");
cudaError_t build_lists(Plan& P, unsigned long long* skipped_total, cudaStream_t st) {
    // up to 8,192 column blocks: 16 keys a thread, two CTAs per SM; up to 16,384: 32 keys a thread;
    // beyond that (n > 4,194,304 with blocks of 256) the lists stay in block order (no early stop)
    const bool wide = P.ncb > ListShape<16>::N;
    auto kern = P.qnorm ? (wide ? k_block_lists<32, true> : k_block_lists<16, true>)
                        : (wide ? k_block_lists<32, false> : k_block_lists<16, false>);
    const size_t smem = (size_t)(wide ? ListShape<32>::N : ListShape<16>::N) * 4;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    kern<<<P.nqb, LIST_T, smem, st>>>(P.qcenter, P.qradius, P.ccenter_f, P.cradius_f, P.nqb, P.ncb, P.d, P.tq,
                                      P.rowmax, P.rm_delta, P.qnorm, P.cnorm, P.norm_only ? 0 : 1, P.lists, P.list_ub, P.counts, P.weight, P.ub_skip, skipped_total);
    note_launch();
    k_block_order<<<1, 1024, 0, st>>>(P.weight, P.nqb, P.ncb, P.order); note_launch();
    k_row_ub<<<(P.n + 255) / 256, 256, 0, st>>>(P.perm, P.n, P.ub_skip, P.row_ub); note_launch();
    return cudaGetLastError();
}

}  // namespace prune
}  // namespace costal
