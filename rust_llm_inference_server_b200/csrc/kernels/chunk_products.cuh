// Small float32 products out of shared memory, for recurrences that take 64 tokens of a request at a time: two-wide FMAs, 8 rows and 4 or 8 columns a
// thread of 128.
#pragma once
#include "common.cuh"
#include <math.h>

namespace chunkprod {
constexpr int CHUNK = 64, LDT = CHUNK + 4;
typedef unsigned long long u64;

__device__ __forceinline__ u64 pack2(float lo, float hi) {
    u64 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void fma2(u64& acc, u64 a, u64 b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
// acc += A^T B over k: 8 rows (ty * 4 + {0..3}, 32 on) and NC columns (tx * 4 + {0..3}, 64 on) a thread.  Two rows share a register pair, as A's
// lie in shared memory, and columns are doubled: with pairs of columns there were twice as many moves (NC 4: 35 instructions a k, 27 so).
// BLOCK > 0: a sum of its own every BLOCK terms, added to acc (with one chain of 128 the outputs were 2.0e-7 off 64 bits, the
// walk's, in shares of 8, are 0.8e-7).
template <int NC> struct Tile {
    u64 v[4][NC];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < NC; ++j) v[i][j] = 0ull;
    }
    // row i (0..7) of the thread's rows, column j
    __device__ __forceinline__ float at(int i, int j) const {
        float lo, hi;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v[i / 2][j]));
        return i & 1 ? hi : lo;
    }
    __device__ __forceinline__ void scale(int i2, float lo, float hi) {      // rows 2 i2 and 2 i2 + 1
        const u64 f = pack2(lo, hi);
#pragma unroll
        for (int j = 0; j < NC; ++j) asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(v[i2][j]) : "l"(f));
    }
    __device__ __forceinline__ void add(const Tile& o) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < NC; ++j) asm("add.rn.f32x2 %0, %0, %1;" : "+l"(v[i][j]) : "l"(o.v[i][j]));
    }
};
// A and B: the thread's first row and column; its other four rows lie FAR on, its columns from the fourth on 64 on.
template <int FAR, int BLOCK, int NC>
__device__ __forceinline__ void rows_product(Tile<NC>& acc, const float* A, int lda, const float* B, int ldb, int K) {
    auto step = [&](int k, Tile<NC>& into) {
        u64 a[4];
        float b[NC];
#pragma unroll
        for (int i = 0; i < 2; ++i) *reinterpret_cast<ulonglong2*>(&a[2 * i]) = *reinterpret_cast<const ulonglong2*>(A + k * lda + i * FAR);
#pragma unroll
        for (int j = 0; j < NC; j += 4) *reinterpret_cast<float4*>(&b[j]) = *reinterpret_cast<const float4*>(B + k * ldb + j * 16);
#pragma unroll
        for (int j = 0; j < NC; ++j) {
            const u64 bb = pack2(b[j], b[j]);
#pragma unroll
            for (int i = 0; i < 4; ++i) fma2(into.v[i][j], a[i], bb);
        }
    };
    if (BLOCK == 0) {
#pragma unroll 8
        for (int k = 0; k < K; ++k) step(k, acc);
        return;
    }
    for (int k0 = 0; k0 < K; k0 += BLOCK) {         // (K is a multiple of BLOCK)
        Tile<NC> part;
        part.clear();
#pragma unroll
        for (int k = 0; k < BLOCK; ++k) step(k0 + k, part);
        acc.add(part);
    }
}

template <int NC, int BLOCK>
__device__ __forceinline__ void product(Tile<NC>& acc, const float* A, int lda, const float* B, int ldb, int K, int ty, int tx) {
    rows_product<32, BLOCK>(acc, A + ty * 4, lda, B + tx * 4, ldb, K);
}

// Place of thread t of 128: 8 x 16 of them, a warp 4 x 8.
__device__ __forceinline__ int thread_row(int t) { return (t >> 6) * 4 + ((t & 31) >> 3); }
__device__ __forceinline__ int thread_col(int t) { return ((t >> 5) & 1) * 8 + (t & 7); }
}  // namespace chunkprod
