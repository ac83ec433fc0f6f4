// The FP32 coarse pass: every (query block × column tile) dot product on the CUDA cores, fused with
// the per-query top-cap selection (crates/costal-core/src/knn.rs:603-660 tiles, :758-787 the
// threshold scan, :791-875 the per-row heaps).
//
//   tile      4 consumer warps own 128 query rows; each thread holds a 16 × 8 register tile (16 queries in
//             groups of 4, columns tx·4+j and 64+tx·4+j), so a warp owns 32 queries and sees all 128
//             columns of a tile for them. Two queries share one paired FP32 FMA (two independent
//             single-rounding FMAs per instruction), so the query pairs come straight from shared
//             memory and only the 8 column values are duplicated in registers. Every score is one
//             FMA chain over the depth in dimension order. The shape is set by shared-memory
//             bandwidth: a 16-byte load costs a warp 2 wavefronts when a half warp shares its address
//             and 4 when it does not, so a depth step costs 16 wavefronts for 64 paired FMAs (128
//             pipe cycles); an 8 × 8 tile costs 12 for 32 (16 with the queries stored twice), as many
//             as the FMAs of 8 warps.
//   pipeline  warp 4 streams column tiles with TMA into a ring of stages (full / empty mbarriers), kc
//             dimensions a stage. The consumer warps never meet at a block barrier: one warp's
//             selection overlaps another's FMAs, and a stage is handed back before its scores are
//             looked at. Two CTAs per SM wherever their shared memory fits. For d_pad ≤ 64 the query
//             operand stays resident; deeper rows stream both operands.
//   select    A row whose tile maximum exceeds its query's τ appends its columns above τ to the query's
//             buffer in shared memory; a buffer about to overflow is cut to its best cap by a warp-wide
//             radix select, and τ rises to the cap-th score. Everything outside the buffer scored ≤ τ
//             when it was seen or cut, and τ only grows: the certificate s_k > τ + ε (k_rescore) covers
//             it. The first tile seeds τ: the cap-th largest of its column-group maxima is reached by
//             cap distinct columns.
//   lists     With prune.cu's lists the rows and columns are in the working order and a CTA visits the
//             column blocks of its list, nearest first: τ is near its final value after the first
//             tiles, and the CTA stops at the first block whose bound is below every query's τ − ε (its
//             columns' coarse scores are ≤ bound + ε, so none could be admitted; later bounds are no
//             larger).
//   walk      Tanimoto selection in the norm order (knn.rs:595-644): a CTA visits its own tile first and
//             then outward on both sides, and leaves a side where the bound that the norms alone give is
//             below every query's τ − ε. O(n) memory at any n, where lists take 12 bytes for every pair of
//             blocks.
//   segments  Few query blocks: the columns are split over gridDim.y CTAs per block and the segments'
//             lists merged per row (k_merge_parts), so that no SM idles in a nearly empty last wave.
//             The segments of a query share their thresholds whenever one of them cuts its buffer.
//
// Every mbarrier wait is bounded (ptx.cuh); a wait that gives up raises timeout_flag, and the producer, the last
// to leave, waits for the loads in flight.

#include <cuda_runtime.h>

#include <algorithm>
#include <math_constants.h>
#include <stdint.h>

#include "common.cuh"
#include "fp32_tile.cuh"
#include "kernels.h"
#include "ptx.cuh"
#include "topk.cuh"

namespace costal {
namespace fp32 {

constexpr int BM = 128;
constexpr int BN = 128;
constexpr int CONS_WARPS = 4;                // consumer warps, 32 queries each
// One warpgroup of consumers and one for the producer (one thread of it works): a launch at 128
// registers a thread, of which the producers give up all but 40 and the consumers take 208. (A lone
// producer warp would be the third warp of a scheduler in two CTAs and cap every thread at 168.)
constexpr int NT = 256;
constexpr int REGS_PRODUCER = 40, REGS_CONSUMER = 208;
static_assert((REGS_PRODUCER + REGS_CONSUMER) * 128 <= NT * 128, "the split stays within the launch's registers");
constexpr int MAX_STAGES = 6;
constexpr size_t SMEM_ONE = 227 * 1024;      // shared memory of a CTA alone on its SM
constexpr size_t SMEM_TWO = 113 * 1024;      // of each of two

struct __align__(8) Bars {
    uint64_t a_full;
    uint64_t full[MAX_STAGES];
    uint64_t empty[MAX_STAGES];
    int c0[MAX_STAGES];  // first column of the stage's tile, −1: no more tiles
    float warp_floor[CONS_WARPS];  // per consumer warp: min over its queries of τ − ε (never decreases)
};

// The cap-th largest of a half warp's 16·R values (R per lane): a bitonic sorting network over the
// 16 lanes, both halves of the warp at once. Out of line: it runs once per row of the first tile.
template <int R>
__device__ __noinline__ float half_kth(float v0, float v1, float v2, float v3, int cap, int lane) {
    float v[4] = {v0, v1, v2, v3};
    const int l = lane & 15;
#pragma unroll
    for (int size = 2; size <= 16 * R; size <<= 1) {
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            if (stride >= 16) {
#pragma unroll
                for (int s = 0; s < R; ++s) {
                    const int t = s ^ (stride >> 4);
                    if (t > s) {
                        const bool desc = ((s * 16 + l) & size) == 0;
                        const float hi = fmaxf(v[s], v[t]), lo = fminf(v[s], v[t]);
                        v[s] = desc ? hi : lo;
                        v[t] = desc ? lo : hi;
                    }
                }
            } else {
#pragma unroll
                for (int s = 0; s < R; ++s) {
                    const float o = __shfl_xor_sync(COSTAL_FULL_MASK, v[s], stride);
                    const bool keep_max = ((l & stride) == 0) == (((s * 16 + l) & size) == 0);
                    v[s] = keep_max ? fmaxf(v[s], o) : fminf(v[s], o);
                }
            }
        }
    }
    float pick = v[0];
#pragma unroll
    for (int s = 1; s < R; ++s)
        if (s == (cap - 1) >> 4) pick = v[s];
    return __shfl_sync(COSTAL_FULL_MASK, pick, (lane & 16) | ((cap - 1) & 15));
}

// Cut one query's buffer (cnt > cap entries) to its best cap, in place, and return the cap-th largest
// score: a warp-wide radix select on order-preserving keys, bit by bit from the highest bit where the
// buffer's keys differ, done as soon as exactly cap keys lie at or above the prefix. Of entries equal
// to the cap-th score the first in the buffer stay.
template <int SLB>
__device__ __noinline__ float cut_buffer(float* bs, uint32_t* bi, int cnt, int cap, int lane) {
    float sc[SLB];
    uint32_t id[SLB], key[SLB];
    uint32_t kmin = 0xffffffffu, kmax = 0u;
#pragma unroll
    for (int s = 0; s < SLB; ++s) {
        const int p = s * 32 + lane;
        const bool v = p < cnt;
        sc[s] = v ? bs[p] : 0.0f;
        id[s] = v ? bi[p] : 0u;
        const uint32_t u = __float_as_uint(sc[s]);
        key[s] = v ? ((u & 0x80000000u) ? ~u : (u | 0x80000000u)) : 0u;  // 0: below every valid key
        if (v) {
            kmin = min(kmin, key[s]);
            kmax = max(kmax, key[s]);
        }
    }
    kmin = __reduce_min_sync(COSTAL_FULL_MASK, kmin);
    kmax = __reduce_max_sync(COSTAL_FULL_MASK, kmax);
    const uint32_t diff = kmin ^ kmax;
    const int top = diff ? 31 - __clz(diff) : -1;
    uint32_t T = top >= 0 ? (kmax & ~((2u << top) - 1u)) : kmax;
    bool whole = false;  // exactly cap keys are ≥ T
    for (int b = top; b >= 0; --b) {
        const uint32_t c = T | (1u << b);
        int n_ge = 0;
#pragma unroll
        for (int s = 0; s < SLB; ++s) n_ge += __popc(__ballot_sync(COSTAL_FULL_MASK, key[s] >= c));
        if (n_ge >= cap) T = c;
        if (n_ge == cap) {
            whole = true;
            break;
        }
    }
    if (whole) {  // the cap-th score is the smallest key at or above the prefix
        uint32_t m = 0xffffffffu;
#pragma unroll
        for (int s = 0; s < SLB; ++s)
            if (key[s] >= T) m = min(m, key[s]);
        T = __reduce_min_sync(COSTAL_FULL_MASK, m);
    }
    int n_gt = 0;
#pragma unroll
    for (int s = 0; s < SLB; ++s) n_gt += __popc(__ballot_sync(COSTAL_FULL_MASK, key[s] > T));
    const unsigned below = (1u << lane) - 1u;
    int eq = 0, kept = 0;
    bool keep[SLB];
    int pos[SLB];
#pragma unroll
    for (int s = 0; s < SLB; ++s) {
        const unsigned meq = __ballot_sync(COSTAL_FULL_MASK, key[s] == T);
        const bool k = key[s] > T || (key[s] == T && eq + __popc(meq & below) < cap - n_gt);
        const unsigned mk = __ballot_sync(COSTAL_FULL_MASK, k);
        keep[s] = k;
        pos[s] = kept + __popc(mk & below);
        eq += __popc(meq);
        kept += __popc(mk);
    }
    __syncwarp();  // every lane has read its entries before any is overwritten
#pragma unroll
    for (int s = 0; s < SLB; ++s) {
        if (keep[s]) {
            bs[pos[s]] = sc[s];
            bi[pos[s]] = id[s];
        }
    }
    __syncwarp();
    return __uint_as_float((T & 0x80000000u) ? (T & 0x7fffffffu) : ~T);
}

struct Args {
    int n;          // columns
    int nq;         // query slots in use
    int cap, bcap, dp, kc, tiles, stages;
    const uint32_t* rows;  // the queries' column ids (NULL: slot q is column q)
    int part_stride;       // > 0: segment lists out, by slot
    const uint32_t* perm;  // working → original row (NULL: identity)
    const uint32_t* lists; // [query blocks][ncb] column blocks, nearest first (NULL: all tiles)
    const float* list_ub;  // their bounds, not increasing (NULL: no early stop)
    const uint32_t* counts;
    const uint32_t* order; // the query block of each CTA (NULL: in order)
    int ncb, epc;          // list stride; 128-column tiles per list entry
    float eps;             // the coarse error bound, rounded up
    const float2* walk;      // norm ranges of the tiles, and what lies after and before them (kernels.h)
    const float2* walk_ends;
    unsigned long long* stopped_total;
    uint32_t* tau_shared;  // with segments: order key of each slot's largest threshold so far
    const float* tfloor;   // by row: no column at or below it can be among the best cap (NULL: none)
    const float2* tnorm;   // Tanimoto: f32 norm and squared norm of every column
    uint32_t* cand_idx;
    float* cand_score;
    float* tau_out;
    unsigned long long* timeout_flag;
};

__device__ __forceinline__ uint32_t okey(float v) {
    const uint32_t u = __float_as_uint(v);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float okey_inv(uint32_t k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// Tanimoto: T > τ > 0 needs a cosine above τ/(1+τ)·(ρ + 1/ρ) ≥ 2τ/(1+τ), ρ the norms' quotient
// (knn.rs:239-283); the factor 1 − 2⁻¹⁶ covers every f32 rounding of T and of this threshold.
__device__ __forceinline__ float tani_cos_floor(float tau) {
    return !(tau > 0.0f)         ? -CUDART_INF_F
           : tau == CUDART_INF_F ? CUDART_INF_F
                                 : 2.0f * __fdividef(tau, 1.0f + tau) * (1.0f - 0x1p-16f);
}

enum Visit {
    IN_ORDER,  // all tiles in order, or the lists of the query blocks in order
    BY_ORDER,  // the lists, the query block of each CTA from P.order
    WALK       // outward in the norm order
};

template <int SLB, bool STREAM, bool TANI, Visit VISIT>
__global__ void __launch_bounds__(NT, 2)
    k_fp32_tiles(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const Args P) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((128 - (smem_u32(smem_raw) & 127)) & 127);
    const int kc = P.kc, bcap = P.bcap, cap = P.cap;
    const uint32_t chunk = (uint32_t)kc * BN * 4;  // one operand's kc dimensions
    const uint32_t stage_bytes = STREAM ? 2 * chunk : chunk;
    unsigned char* a_res = smem;                                          // resident query operand
    unsigned char* ring = STREAM ? smem : smem + (size_t)P.dp * BM * 4;   // stages × (A chunk, B chunk) or × B chunk
    float* buf_s = reinterpret_cast<float*>(ring + (size_t)P.stages * stage_bytes);  // [BM][bcap]
    uint32_t* buf_i = reinterpret_cast<uint32_t*>(buf_s + BM * bcap);
    int* cnt_s = reinterpret_cast<int*>(buf_i + BM * bcap);
    float* tau_s = reinterpret_cast<float*>(cnt_s + BM);
    int* own_s = reinterpret_cast<int*>(tau_s + BM);  // the query's own column, −1: no query
    Bars* bars = reinterpret_cast<Bars*>(own_s + BM);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // (a template parameter: with the choice made at run time the whole kernel was 7 % slower)
    const int qb = VISIT == BY_ORDER ? (int)P.order[blockIdx.x] : (int)blockIdx.x, q0 = qb * BM;
    const int nch = (P.dp + kc - 1) / kc;
    if (tid == 0) {
        mbar_init(&bars->a_full, 1);
        for (int s = 0; s < P.stages; ++s) {
            mbar_init(&bars->full[s], 1);
            mbar_init(&bars->empty[s], CONS_WARPS);
        }
        for (int w = 0; w < CONS_WARPS; ++w) bars->warp_floor[w] = -CUDART_INF_F;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int q = tid; q < BM; q += NT) {
        const int own = q0 + q < P.nq ? (P.rows ? (int)P.rows[q0 + q] : q0 + q) : -1;
        own_s[q] = own;
        cnt_s[q] = 0;
        tau_s[q] = own < 0 ? CUDART_INF_F : (P.tfloor ? P.tfloor[own] : -CUDART_INF_F);  // no query: never admits
    }
    __syncthreads();

    if (warp >= CONS_WARPS) {
        // ------------------------------------------------------------------ TMA producer
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS_PRODUCER));
        if (tid != CONS_WARPS * 32) return;
        if (!STREAM) {
            mbar_expect_tx(&bars->a_full, (uint32_t)P.dp * BM * 4);
            for (int t = 0; t < P.dp; t += kc) tma_load_2d(a_res + (size_t)t * BM * 4, &map_a, q0, t, &bars->a_full);
        }
        int s = 0;
        uint32_t ph = 1;
        auto next_stage = [&]() {
            if (++s == P.stages) {
                s = 0;
                ph ^= 1u;
            }
        };
        auto wait_empty = [&]() -> bool {
            if (mbar_wait(&bars->empty[s], ph, P.timeout_flag, true)) return true;
            drain_ring(bars->full, P.stages, s, ph);
            if (!STREAM) mbar_drain(&bars->a_full, 0);
            return false;
        };
        auto send_tile = [&](int c0) -> bool {
            for (int ch = 0; ch < nch; ++ch) {
                if (!wait_empty()) return false;
                unsigned char* dst = ring + (size_t)s * stage_bytes;
                bars->c0[s] = c0;
                mbar_expect_tx(&bars->full[s], stage_bytes);
                if (STREAM) tma_load_2d(dst + chunk, &map_a, q0, ch * kc, &bars->full[s]);
                tma_load_2d(dst, &map_b, c0, ch * kc, &bars->full[s]);
                next_stage();
            }
            return true;
        };
        const int seg = (int)blockIdx.y, segs = (int)gridDim.y;
        if (VISIT == WALK) {  // the segment's steps of the walk: every segs-th one
            // Steps alternate between the sides while both last, own tile first, so that a step's tile needs no
            // other step's bound (chosen by bound, a segment had to follow all steps: 3 to 7 % slower). A side
            // ends at its first tile whose bound is below the floors: later ones are no larger.
            const float2 nq = P.walk[qb];
            const int nl = qb + 1, nr = P.tiles - nl, both = 2 * min(nl, nr);
            bool l_out = false, r_out = false;
            unsigned out = 0;
            for (int e = seg; e < P.tiles; e += segs) {
                const bool left = e < both ? !(e & 1) : nl > nr;
                const int i = e < both ? e >> 1 : e - both / 2, t = left ? qb - i : nl + i;
                if (!(left ? l_out : r_out)) {
                    const float2 ends = P.walk_ends[t];
                    const float ub = tani_ub_f32(1.0f, nq, left ? make_float2(0.0f, ends.y) : make_float2(ends.x, CUDART_INF_F));
                    volatile float* wf = bars->warp_floor;  // may be stale, i.e. lower: that only delays the stop
                    if (!(ub < fminf(fminf(wf[0], wf[1]), fminf(wf[2], wf[3])))) {
                        if (!send_tile(t * BN)) return;
                        continue;
                    }
                    (left ? l_out : r_out) = true;
                }
                if ((l_out && r_out) || e >= both) {  // only tiles of a side that has ended are left
                    out += (unsigned)((P.tiles - e + segs - 1) / segs);
                    break;
                }
                ++out;
            }
            if (P.stopped_total && out) atomicAdd(P.stopped_total, (unsigned long long)out);
        } else if (P.lists) {  // the segment's list entries: every segs-th one
            const uint32_t* list = P.lists + (size_t)qb * P.ncb;
            const float* ub = P.list_ub ? P.list_ub + (size_t)qb * P.ncb : nullptr;
            const int count = min((int)P.counts[qb], P.ncb);
            const int limit_c = P.tiles * BN;
            for (int e = seg; e < count; e += segs) {
                if (ub) {
                    volatile float* wf = bars->warp_floor;  // may be stale, i.e. lower: that only delays the stop
                    if (ub[e] < fminf(fminf(wf[0], wf[1]), fminf(wf[2], wf[3]))) {
                        if (P.stopped_total) atomicAdd(P.stopped_total, (unsigned long long)((count - e + segs - 1) / segs));
                        break;
                    }
                }
                for (int h = 0; h < P.epc; ++h) {
                    const long long c0 = ((long long)list[e] * P.epc + h) * BN;
                    if (c0 < limit_c && !send_tile((int)c0)) return;
                }
            }
        } else {
            const int tps = (P.tiles + segs - 1) / segs;
            for (int t = seg * tps; t < min(P.tiles, (seg + 1) * tps); ++t)
                if (!send_tile(t * BN)) return;
        }
        if (!wait_empty()) return;
        bars->c0[s] = -1;
        mbar_arrive(&bars->full[s]);  // completes the phase without data (release)
        return;
    }

    // ---------------------------------------------------------------------- consumers
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS_CONSUMER));
    const int tx = lane & 15, ty = 2 * warp + (lane >> 4);
    auto qi_at = [&](int i, int y) { return tile_row(i, y); };  // query i of thread row y
    auto cj_of = [&](int j) { return tile_col(j, tx); };
    const int limit = cap + (bcap - cap) * 3 / 4;
    if (!STREAM && !mbar_wait(&bars->a_full, 0, P.timeout_flag, false)) return;
    int s = 0;
    uint32_t ph = 0;
    for (bool first = true;; first = false) {
        unsigned long long acc[8][8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[i][j] = 0ull;
        int c0 = 0;
        for (int ch = 0; ch < nch; ++ch) {
            if (!mbar_wait(&bars->full[s], ph, P.timeout_flag, false)) return;
            c0 = *reinterpret_cast<volatile int*>(&bars->c0[s]);
            if (c0 < 0) break;
            const unsigned char* st = ring + (size_t)s * stage_bytes;
            const ulonglong2* A = reinterpret_cast<const ulonglong2*>(STREAM ? st + chunk : a_res + (size_t)ch * chunk);
            const float4* B = reinterpret_cast<const float4*>(st);
#pragma unroll 1
            for (int k = 0; k < kc; k += 8) fma8(A + k * 32, B + k * 32, tx, ty, acc);
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->empty[s]);
            if (++s == P.stages) {
                s = 0;
                ph ^= 1u;
            }
        }
        if (c0 < 0) break;
        auto score = [&](int i, int j) { return tile_score(acc, i, j); };
        // rows whose tile maximum is above their threshold (Tanimoto: above the cosine that threshold needs)
        unsigned m = 0;
        if (!first) {
#pragma unroll
            for (int i4 = 0; i4 < 4; ++i4) {
                const float4 tr = *reinterpret_cast<const float4*>(tau_s + i4 * 32 + ty * 4);
                const float t4[4] = {tr.x, tr.y, tr.z, tr.w};
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int i = i4 * 4 + u;
                    const float top = max3(max3(score(i, 0), score(i, 1), score(i, 2)),
                                           max3(score(i, 3), score(i, 4), score(i, 5)), fmaxf(score(i, 6), score(i, 7)));
                    m |= (top > (TANI ? tani_cos_floor(t4[u]) : t4[u]) ? 1u : 0u) << i;
                }
            }
            m = __reduce_or_sync(COSTAL_FULL_MASK, m);
            if (m == 0) continue;
        } else {
            m = 0xffffu;
        }
        // a tile with the queries' own columns or the padding: those columns never count
        const bool edge = P.rows != nullptr || c0 + BN > P.n || c0 == q0;
        // (One copy of this path, the row's scores picked by a jump: unrolled over the rows its code
        // overflows the instruction cache, 4.8 against 1.7 ms at 20,000 × 32.)
#pragma unroll 1
        while (m) {
            const int i = __ffs(m) - 1;  // warp-uniform
            m &= m - 1;
            float sv[8];
            switch (i) {
#define COSTAL_ROW(r)                                     \
    case r:                                               \
        _Pragma("unroll") for (int j = 0; j < 8; ++j) sv[j] = score(r, j); \
        break;
                COSTAL_ROW(0) COSTAL_ROW(1) COSTAL_ROW(2) COSTAL_ROW(3) COSTAL_ROW(4) COSTAL_ROW(5) COSTAL_ROW(6)
                COSTAL_ROW(7) COSTAL_ROW(8) COSTAL_ROW(9) COSTAL_ROW(10) COSTAL_ROW(11) COSTAL_ROW(12)
                COSTAL_ROW(13) COSTAL_ROW(14)
                default: COSTAL_ROW(15)
#undef COSTAL_ROW
            }
            const int qi = qi_at(i, ty), own = own_s[qi];
            float* bs = buf_s + qi * bcap;
            uint32_t* bi = buf_i + qi * bcap;
            float tau = tau_s[qi];
            const float2 qn = TANI && own >= 0 ? P.tnorm[own] : make_float2(0.f, 0.f);
            const float cf = TANI && !first ? tani_cos_floor(tau) : -CUDART_INF_F;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int col = c0 + cj_of(j);
                if (TANI) sv[j] = sv[j] > cf ? tani_coarse_f32(sv[j], qn, col < P.n ? P.tnorm[col] : make_float2(0.f, 0.f))
                                             : -CUDART_INF_F;
                if (edge && (col >= P.n || col == own)) sv[j] = -CUDART_INF_F;
            }
            if (first && cap <= 64) {
                // the seed: the cap-th largest of 32 maxima of 4 columns (cap ≤ 32), or of 64 of 2
                float t0;
                if (cap <= 32)
                    t0 = half_kth<2>(fmaxf(max3(sv[0], sv[1], sv[2]), sv[3]), fmaxf(max3(sv[4], sv[5], sv[6]), sv[7]), 0.f,
                                     0.f, cap, lane);
                else
                    t0 = half_kth<4>(fmaxf(sv[0], sv[1]), fmaxf(sv[2], sv[3]), fmaxf(sv[4], sv[5]), fmaxf(sv[6], sv[7]),
                                     cap, lane);
                if (t0 > -CUDART_INF_F) tau = fmaxf(tau, nextafterf(t0, -CUDART_INF_F));
                if (tx == 0) tau_s[qi] = tau;
            }
            unsigned pend = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) pend |= (sv[j] > tau ? 1u : 0u) << j;
            while (__any_sync(COSTAL_FULL_MASK, pend != 0)) {
                int pos = pend ? atomicAdd(&cnt_s[qi], __popc(pend)) : 0;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    if (pend >> j & 1u) {
                        if (pos < bcap) {
                            bs[pos] = sv[j];
                            bi[pos] = (uint32_t)(c0 + cj_of(j));
                            pend &= ~(1u << j);
                        }
                        ++pos;
                    }
                }
                __syncwarp();
                const int c = cnt_s[qi];
                const unsigned over = __ballot_sync(COSTAL_FULL_MASK, c > limit);
                if (over) {
#pragma unroll 1
                    for (int h = 0; h < 2; ++h) {
                        if (!(over >> (16 * h) & 1u)) continue;
                        const int qh = qi_at(i, 2 * warp + h);
                        float T = cut_buffer<SLB>(buf_s + qh * bcap, buf_i + qh * bcap,
                                                  min(bcap, __shfl_sync(COSTAL_FULL_MASK, c, 16 * h)), cap, lane);
                        if (lane == 0) {
                            if (P.tau_shared) {
                                const uint32_t k = okey(T);
                                T = okey_inv(max(k, atomicMax(&P.tau_shared[q0 + qh], k)));
                            }
                            cnt_s[qh] = cap;
                            tau_s[qh] = T;
                        }
                    }
                    __syncwarp();
                    tau = tau_s[qi];
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (!(sv[j] > tau)) pend &= ~(1u << j);
                }
            }
        }
        __syncwarp();  // every lane sees the thresholds before the next tile's test
        if (VISIT == WALK || P.list_ub) {  // the warp's floor for the producer's stop test (signed-int order of the f32)
            int key = __float_as_int(__fsub_rd(tau_s[qi_at(lane & 15, ty)], P.eps));
            key = __reduce_min_sync(COSTAL_FULL_MASK, key >= 0 ? key : key ^ 0x7fffffff);
            if (lane == 0)
                *reinterpret_cast<volatile float*>(&bars->warp_floor[warp]) = __int_as_float(key >= 0 ? key : key ^ 0x7fffffff);
        }
    }

    // the warp's 32 queries out: by row, or by slot into the segment's part
    __syncwarp();
#pragma unroll 1
    for (int e = 0; e < 32; ++e) {
        const int qi = qi_at(e & 15, 2 * warp + (e >> 4)), own = own_s[qi];
        if (own < 0) continue;
        int c = min(bcap, cnt_s[qi]);
        float tau = tau_s[qi];
        if (c > cap) {
            tau = fmaxf(tau, cut_buffer<SLB>(buf_s + qi * bcap, buf_i + qi * bcap, c, cap, lane));
            c = cap;
        }
        const size_t row = P.part_stride ? (size_t)blockIdx.y * P.part_stride + q0 + qi
                                         : (size_t)(P.perm ? P.perm[own] : (uint32_t)own);
        for (int p = lane; p < cap; p += 32) {
            const uint32_t col = p < c ? buf_i[qi * bcap + p] : 0xffffffffu;
            P.cand_idx[row * cap + p] = p < c && P.perm ? P.perm[col] : col;
            P.cand_score[row * cap + p] = p < c ? buf_s[qi * bcap + p] : -CUDART_INF_F;
        }
        if (lane == 0) P.tau_out[row] = tau;
    }
}

// The transposed copy in working order: out[t][w] = xsR[perm[w]][t] (xsR row-major [n][d]), zero for w ≥ n
// and t ≥ d: a CTA per 128 rows, staged through shared memory so that whole rows are read and both
// sides are coalesced.
__global__ void __launch_bounds__(256) k_work_cols(const float* __restrict__ xsR, const uint32_t* __restrict__ perm, int n,
                                                   int np, int d, int dp, float* __restrict__ out) {
    extern __shared__ float tile[];  // [BM][d + 1]
    const int w0 = blockIdx.x * BM, rows = min(BM, n - w0);
    for (int e = threadIdx.x; e < rows * d; e += 256)
        tile[(e / d) * (d + 1) + e % d] = xsR[(size_t)perm[w0 + e / d] * d + e % d];
    __syncthreads();
    for (int e = threadIdx.x; e < dp * BM; e += 256) {
        const int t = e / BM, r = e % BM;
        out[(size_t)t * np + w0 + r] = r < rows && t < d ? tile[r * (d + 1) + t] : 0.0f;
    }
}

// The listed queries' columns of xsT, side by side: out[t][q] = value t of row rows[q], zero for
// q ≥ nq; mp = the slots rounded up to a whole block.
__global__ void k_gather_cols(const float* __restrict__ xsT, int np, int dp, const uint32_t* __restrict__ rows, int nq,
                              int mp, float* __restrict__ out) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= mp) return;
    const uint32_t c = q < nq ? rows[q] : 0u;
    for (int t = blockIdx.y; t < dp; t += gridDim.y) out[(size_t)t * mp + q] = q < nq ? xsT[(size_t)t * np + c] : 0.0f;
}

// The rows' f32 norm and squared norm from the f64 norms (knn.rs:207-212 rounds ‖x‖² to f32), in working order.
__global__ void k_tani_norms(const double* __restrict__ norms, int n, const uint32_t* __restrict__ perm,
                             float2* __restrict__ tnorm) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double a = norms[perm ? perm[i] : (uint32_t)i];
        tnorm[i] = make_float2((float)a, (float)(a * a));
    }
}

// One warp per listed row: the union of its segments' lists (segs · cap entries) as (score desc,
// index asc) keys, 256 at a time: after each warp sort the first cap positions hold the best so far
// and the other 256 − cap take the next entries. The best cap go to the row's candidates, and τ is
// the cap-th score (≥ every segment's own τ, since a full segment list holds cap entries at or above
// it), or the row's floor when the segments hold fewer than cap together.
__global__ void k_merge_parts(const uint32_t* __restrict__ qlist, int count, int segs, int cap,
                              const uint32_t* __restrict__ part_idx, const float* __restrict__ part_score,
                              const float* __restrict__ tfloor, int lstride, uint32_t* __restrict__ cand_idx,
                              float* __restrict__ cand_score, float* __restrict__ tau_out) {
    const int lane = threadIdx.x & 31;
    const int r = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (r >= count) return;
    const int total = segs * cap;
    auto load = [&](int e) {
        if (e >= total) return PAD_KEY;
        const size_t o = ((size_t)(e / cap) * count + r) * cap + e % cap;
        return order_key(part_score[o], part_idx[o]);
    };
    uint64_t key[8];
#pragma unroll
    for (int s = 0; s < 8; ++s) key[s] = load(s * 32 + lane);
    warp_sort_keys<8>(key, lane);
    for (int next = 256; next < total; next += 256 - cap) {  // warp-uniform
#pragma unroll
        for (int s = 0; s < 8; ++s) {
            const int p = s * 32 + lane;
            if (p >= cap) key[s] = load(next + p - cap);
        }
        warp_sort_keys<8>(key, lane);
    }
    const uint32_t q = qlist ? qlist[r] : (uint32_t)r;
    uint64_t kth = 0;
#pragma unroll
    for (int s = 0; s < 8; ++s) {
        const int p = s * 32 + lane;
        if (p < cap) {
            cand_idx[(size_t)q * lstride + p] = key_index(key[s]);
            cand_score[(size_t)q * lstride + p] = key_score(key[s]);
        }
        if (s == (cap - 1) >> 5) kth = key[s];
    }
    const uint64_t t = __shfl_sync(COSTAL_FULL_MASK, kth, (cap - 1) & 31);
    // with fewer than cap candidates in all segments together, the row's floor still bounds the rest
    if (lane == 0) tau_out[q] = fmaxf(key_score(t), tfloor ? tfloor[q] : -CUDART_INF_F);
}

// The launch shape for a depth and a candidate count: the query operand resident or streamed, the
// buffer's entries, the dimensions and number of the ring's stages, CTAs per SM. Two CTAs per SM with
// buffers of cap + 32 entries if they fit, else down to cap + 16. Where a resident query operand leaves room
// for one only (about 48 candidates and more at d = 64): with more query blocks than SMs (many) the query
// operand is streamed so that two fit (60,000 × 64 Gaussian rows, k = 30 20.0 -> 16.8 ms, Tanimoto 29.6 ->
// 22.6); with fewer, one wave of single CTAs starts cold once for a query block where two CTAs would be two
// halves of one (8,000 × 48, k = 40 1.15 with one, 1.41 with two; 16,383 × 48 2.35 and 3.12).
struct Shape {
    bool stream;
    int bcap, kc, stages, ctas;
    size_t smem;
};

static Shape shape_of(int dp, int cap, bool many) {
    for (int ctas = 2; ctas >= 1; --ctas)
        for (int stream = dp > 64; stream < (dp > 64 || (ctas == 2 && many) ? 2 : 1); ++stream)
            for (int extra = 32; extra >= 16; extra -= 8) {
                Shape s{};
                s.ctas = ctas;
                s.stream = stream;
                s.bcap = (cap + extra + 3) / 4 * 4;
                const size_t lim = ctas == 2 ? SMEM_TWO : SMEM_ONE;
                const size_t fixed = 128 + (size_t)BM * s.bcap * 8 + BM * 12 + sizeof(Bars) + (stream ? 0 : (size_t)dp * BM * 4);
                if (fixed >= lim) continue;
                // the deepest stage of which two fit (whole tiles), else three
                const int most = stream ? 16 : dp;
                for (int kc = most; kc >= 8; kc -= 8) {
                    if (!stream && dp % kc) continue;
                    const size_t per = (size_t)kc * BN * 4 * (stream ? 2 : 1);
                    const int stages = (int)std::min<size_t>(MAX_STAGES, (lim - fixed) / per);
                    if (stages < (kc == dp ? 2 : 3)) continue;
                    s.kc = kc;
                    s.stages = stages;
                    s.smem = fixed + stages * per;
                    return s;
                }
            }
    return Shape{};
}

// [rows][cols] f32 with boxes of box_cols × box_rows.
static bool make_map(CUtensorMap* m, const void* base, size_t cols, int rows, int box_cols, int box_rows) {
    auto fn = tensor_map_encode_fn();
    if (!fn) return false;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)cols * 4};
    cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Column segments for nq queries against `tiles` column tiles: the number whose last wave of CTAs
// (`slots` at a time) ends first, a CTA costing its tiles plus `start` tiles' worth of time for loading
// its queries, seeding, its first admissions (they grow with cap; next to a deep tile they are little) and
// writing its lists (and the merge reading one more list).
static int segments(int nq, int tiles, int dp, int cap, int slots) {
    const int blocks = (nq + BM - 1) / BM;
    const double start = 1.0 + 64.0 / dp + cap / 32.0 * std::min(1.0, 64.0 / dp);
    int best = 1;
    double best_t = 1e300;
    for (int s = 1; s <= std::min(256, tiles); ++s) {
        const int tps = (tiles + s - 1) / s;
        if ((tiles + tps - 1) / tps != s) continue;  // an empty segment
        const double waves = (double)(((long long)blocks * s + slots - 1) / slots);
        const double t = waves * (tps + start) * (1.0 + 1e-3 * s);
        if (t < best_t * 0.98) {
            best_t = t;
            best = s;
        }
    }
    return best;
}

static Shape shape_of(const Fp32Job& J, int sm_count) {
    return shape_of(J.dp, J.cap, (J.nq + BM - 1) / BM > sm_count);
}

static inline size_t al256(size_t b) { return (b + 255) & ~(size_t)255; }

}  // namespace fp32

namespace fp32 {
struct Ws {
    float* a;             // the listed queries' operand
    uint32_t* part_idx;   // with segments: their lists, and the shared thresholds
    float* part_score;
    float* part_tau;
    uint32_t* tau_shared;
    size_t bytes;
};
static Ws carve(void* base, int dp, int cap, bool listed, int nq, int segs) {
    const size_t mp = (size_t)(nq + BM - 1) / BM * BM;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char* p = static_cast<char*>(base) + off;
        off += al256(bytes);
        return p;
    };
    Ws w{};
    w.a = reinterpret_cast<float*>(take(listed ? (size_t)dp * mp * 4 : 0));
    const size_t per = segs > 1 ? (size_t)segs * nq : 0;
    w.part_idx = reinterpret_cast<uint32_t*>(take(per * cap * 4));
    w.part_score = reinterpret_cast<float*>(take(per * cap * 4));
    w.part_tau = reinterpret_cast<float*>(take(per * 4));
    w.tau_shared = reinterpret_cast<uint32_t*>(take(segs > 1 ? mp * 4 : 0));
    w.bytes = off;
    return w;
}
}  // namespace fp32

cudaError_t launch_work_cols(const float* xsR, const uint32_t* perm, int n, int np, int d, int dp, float* xsW,
                             cudaStream_t st) {
    fp32::k_work_cols<<<np / fp32::BM, 256, (size_t)fp32::BM * (d + 1) * 4, st>>>(xsR, perm, n, np, d, dp, xsW);
    note_launch();
    return cudaGetLastError();
}

// With lists (and in the walk) the CTAs' lengths differ and fill each other's gaps: two waves of them are enough (every
// segment starts cold: 100,003 × 15 Tanimoto 5.1 ms with 1 segment, 6.8 with 3), and one wave of single CTAs,
// whose start nothing hides (18,000 × 64 Tanimoto, k = 30 5.17 -> 4.34). A segment keeps at least 24 entries (its
// stop comes a ring of stages after its thresholds have risen).
static int segs_of(const Fp32Job& J, const fp32::Shape& sh, int sm_count) {
    const int blocks = (J.nq + fp32::BM - 1) / fp32::BM, slots = sm_count * sh.ctas;
    if (!J.lists && !J.walk) return fp32::segments(J.nq, J.np / fp32::BN, J.dp, J.cap, slots);
    return std::max(1, std::min(sh.ctas == 1 ? slots / blocks : (2 * slots + blocks - 1) / blocks, (J.walk ? blocks : J.ncb) / 24));
}

size_t coarse_fp32_ws_bytes(const Fp32Job& J, int sm_count) {
    const fp32::Shape sh = fp32::shape_of(J, sm_count);
    const int segs = segs_of(J, sh, sm_count);
    return fp32::carve(nullptr, J.dp, J.cap, J.rows != nullptr, J.nq, segs).bytes;
}

// The lists of `segs` column segments (segs × count × cap entries, τ: segs × count) merged per row.
static cudaError_t launch_merge_parts(const uint32_t* rows, int count, int segs, int cap, const uint32_t* part_idx,
                               const float* part_score, const float* tfloor, uint32_t* cand_idx, float* cand_score,
                               float* tau, cudaStream_t st) {
    fp32::k_merge_parts<<<(count + 7) / 8, 256, 0, st>>>(rows, count, segs, cap, part_idx, part_score, tfloor, cap,
                                                          cand_idx, cand_score, tau);
    note_launch();
    return cudaGetLastError();
}

// The re-run's floor for each listed row, from the tensor-core pass it follows: when that pass kept a
// full list of cap candidates above its threshold τ, their exact cosines are ≥ τ − E_i, so the row's
// cap-th FP32 score is ≥ τ − E_i − ε; below that no column can be among the best cap (rounded down).
__global__ void k_rerun_floor(const uint32_t* __restrict__ rows, const unsigned* __restrict__ count, int cap,
                              const float* __restrict__ tau, const float* __restrict__ cand_score,
                              const double* __restrict__ row_eps, double eps, float* __restrict__ tfloor) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= (int)*count) return;
    const uint32_t i = rows[r];
    const bool full = cand_score[(size_t)i * cap + cap - 1] > -CUDART_INF_F;
    tfloor[i] = full ? __double2float_rd(__dsub_rd(__dsub_rd((double)tau[i], row_eps[i]), eps)) : -CUDART_INF_F;
}

cudaError_t launch_rerun_floor(const uint32_t* rows, const unsigned* count, int nmax, int cap, const float* tau,
                               const float* cand_score, const double* row_eps, double eps, float* tfloor,
                               cudaStream_t st) {
    if (nmax <= 0) return cudaSuccess;
    k_rerun_floor<<<(nmax + 255) / 256, 256, 0, st>>>(rows, count, cap, tau, cand_score, row_eps, eps, tfloor);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_coarse_fp32(const Fp32Job& J, void* ws, int sm_count, cudaStream_t st) {
    using namespace fp32;
    if (J.nq <= 0) return cudaSuccess;
    const Shape sh = shape_of(J, sm_count);
    if (sh.stages < 2 || (J.walk && !J.norms)) return cudaErrorInvalidValue;
    const int mp = (J.nq + BM - 1) / BM * BM, tiles = J.np / BN;
    const int segs = segs_of(J, sh, sm_count);
    const Ws w = carve(ws, J.dp, J.cap, J.rows != nullptr, J.nq, segs);
    cudaError_t e;
    if (J.norms) {
        k_tani_norms<<<std::min((J.n + 255) / 256, 1024), 256, 0, st>>>(J.norms, J.n, J.perm, J.tnorm); note_launch();
    }
    if (J.rows) {
        k_gather_cols<<<dim3(mp / BM, std::min(J.dp, 64)), BM, 0, st>>>(J.xsT, J.np, J.dp, J.rows, J.nq, mp, w.a);
        note_launch();
    }
    if (segs > 1 && (e = cudaMemsetAsync(w.tau_shared, 0, (size_t)mp * 4, st)) != cudaSuccess) return e;
    CUtensorMap ma, mb;
    if (!make_map(&ma, J.rows ? w.a : J.xsT, J.rows ? mp : J.np, J.dp, BM, sh.kc) ||
        !make_map(&mb, J.xsT, J.np, J.dp, BN, sh.kc))
        return cudaErrorInvalidValue;
    Args P{};
    P.n = J.n;
    P.nq = J.nq;
    P.cap = J.cap;
    P.bcap = sh.bcap;
    P.dp = J.dp;
    P.kc = sh.kc;
    P.tiles = tiles;
    P.stages = sh.stages;
    P.rows = J.rows;
    P.perm = J.perm;
    P.lists = J.lists;
    P.list_ub = J.lists ? J.list_ub : nullptr;
    P.counts = J.counts;
    // longest lists first (161,443 × 32 12.7 -> 11.5 ms); with segments the blocks' segments fill the last
    // wave already, and the order costs (30,000 × 15 1.2 -> 1.4 ms)
    P.order = J.lists && segs == 1 ? J.order : nullptr;
    P.ncb = J.ncb;
    P.epc = J.list_cb / BN;
    P.eps = J.eps;
    P.walk = J.walk;
    P.walk_ends = J.walk_ends;
    P.stopped_total = J.stopped_total;
    P.part_stride = segs > 1 ? J.nq : 0;
    P.tau_shared = segs > 1 ? w.tau_shared : nullptr;
    P.tfloor = J.tfloor;
    P.tnorm = J.norms ? J.tnorm : nullptr;
    P.cand_idx = segs > 1 ? w.part_idx : J.cand_idx;
    P.cand_score = segs > 1 ? w.part_score : J.cand_score;
    P.tau_out = segs > 1 ? w.part_tau : J.tau;
    P.timeout_flag = J.timeout_flag;
    const int slb = (sh.bcap + 31) / 32;
#define COSTAL_T(S, ST, V) (J.norms ? k_fp32_tiles<S, ST, true, V> : k_fp32_tiles<S, ST, false, V>)
#define COSTAL_V(S, ST) \
    (J.walk ? k_fp32_tiles<S, ST, true, WALK> : P.order ? COSTAL_T(S, ST, BY_ORDER) : COSTAL_T(S, ST, IN_ORDER))
#define COSTAL_K(S) (sh.stream ? COSTAL_V(S, true) : COSTAL_V(S, false))
    auto kern = slb <= 2 ? COSTAL_K(2) : slb == 3 ? COSTAL_K(3) : COSTAL_K(5);
#undef COSTAL_T
#undef COSTAL_V
#undef COSTAL_K
    if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh.smem)) != cudaSuccess) return e;
    kern<<<dim3(mp / BM, segs), NT, sh.smem, st>>>(ma, mb, P); note_launch();
    if (segs > 1)
        return launch_merge_parts(J.rows ? J.rows : J.perm, J.nq, segs, J.cap, w.part_idx, w.part_score, J.tfloor, J.cand_idx, J.cand_score,
                                  J.tau, st);
    return cudaGetLastError();
}

int coarse_dpad(int d) { return d <= 64 ? ((d < 1 ? 1 : d) + 7) / 8 * 8 : (d + 3) / 4 * 4; }

bool coarse_fp32_holds(int dp, int cap) { return cap <= 128 && fp32::shape_of(dp, cap, false).stages >= 2; }

}  // namespace costal
