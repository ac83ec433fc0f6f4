// The 16 × 8 FP32 register tile of the CUDA-core kernels: a warp's two half warps hold 16 rows each (in
// four groups of 4: row i of thread row ty is (i / 4)·32 + 4·ty + i mod 4 of 128), its 16 lane columns
// tx·4 + j and 64 + tx·4 + j of 128. Rows are paired in the paired FP32 FMA, so every score is one
// single-rounding FMA chain over the depth in order.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace costal {
namespace fp32 {

__device__ __forceinline__ unsigned long long ffma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ float lo_of(unsigned long long r) { return __uint_as_float((uint32_t)r); }
__device__ __forceinline__ float hi_of(unsigned long long r) { return __uint_as_float((uint32_t)(r >> 32)); }
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

__device__ __forceinline__ unsigned long long twice(float x) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
    return r;
}

// 8 depth steps of the register tile. A: [t][128] queries, B: [t][128] columns, 16 bytes an element
// here; acc[p][j] holds queries 2p and 2p + 1 of the thread's 16 and column j of its 8.
__device__ __forceinline__ void fma8(const ulonglong2* A, const float4* B, int tx, int ty,
                                     unsigned long long (&acc)[8][8]) {
#pragma unroll
    for (int t = 0; t < 8; ++t) {
        const ulonglong2 a0 = A[t * 32 + ty], a1 = A[t * 32 + 8 + ty], a2 = A[t * 32 + 16 + ty], a3 = A[t * 32 + 24 + ty];
        const float4 b0 = B[t * 32 + tx], b1 = B[t * 32 + 16 + tx];
        const unsigned long long a[8] = {a0.x, a0.y, a1.x, a1.y, a2.x, a2.y, a3.x, a3.y};
        const float b[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const unsigned long long bb = twice(b[j]);
#pragma unroll
            for (int p = 0; p < 8; ++p) acc[p][j] = ffma2(a[p], bb, acc[p][j]);
        }
    }
}

__device__ __forceinline__ int tile_row(int i, int ty) { return (i >> 2) * 32 + ty * 4 + (i & 3); }
__device__ __forceinline__ int tile_col(int j, int tx) { return j < 4 ? tx * 4 + j : 64 + tx * 4 + (j - 4); }
// The score of row i and column j of the tile's accumulators.
__device__ __forceinline__ float tile_score(const unsigned long long (&acc)[8][8], int i, int j) {
    return i & 1 ? hi_of(acc[i >> 1][j]) : lo_of(acc[i >> 1][j]);
}

}  // namespace fp32
}  // namespace costal
