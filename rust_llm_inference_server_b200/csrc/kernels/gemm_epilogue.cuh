// What the epilogue warps of the tcgen05 products do with 32 consecutive float32 sums of one row.
#pragma once
#include "common.cuh"
#include "mma_utils.cuh"
#include <math.h>

namespace tc {

// Parameters of the gated epilogue with clipping (EPI 3): g' sigmoid(slope g') (u' + shift) with g' = min(g,
// limit) and u' = clamp(u, -limit, limit); limit +inf clips nothing; slope +inf: max(g', 0) (u' + shift); the gate's
// argument is g' + cubic g'^3.  bias (float32, one
// a column; null: none) is added to g and u first.
struct GluParams {
    float slope, limit, shift;
    const float* bias;
    float cubic;
};

// The bias of 32 columns, one a lane (requested before the sums are read), and its addition to every lane's row of sums.
__device__ __forceinline__ float bias_of_lane(const GluParams& gp, int col, int lane, int N) {
    return gp.bias != nullptr && col + lane < N ? gp.bias[col + lane] : 0.f;
}
__device__ __forceinline__ void add_bias32(uint32_t (&r)[32], float bias) {
#pragma unroll
    for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) + __shfl_sync(0xffffffffu, bias, i));
}

// EPI 0: bf16 y [M, N].  EPI 1: SwiGLU over a gate|up matrix whose rows are interleaved in blocks of
// 4 (columns 8 t .. 8 t + 3 gate, 8 t + 4 .. 8 t + 7 up), y [M, N / 2] bf16.  EPI 2: float32 y [M, N].
// EPI 3: the layout of EPI 1 with the clipped gating of GluParams.
// Gates are the function of `glu_gate` to the last bit (expf and a division; gelu's form without limits excepted), so that a token
// gets the same numbers here, in the streaming products of a decode step and in the gating kernels.  They matter: a tile has
// 32,768 of them, and on four warps they took longer than its products (a scheduler runs one warp of the epilogue, so nothing
// hides a chain of 40 instructions).  With eight epilogue warps and one form a launch: 4,096 rows, K 512, N 8192: SwiGLU 76 -> 47 us,
// clipped 90 -> 58 us; 2,048 rows, K 2048, N 16384: 104 -> 101 and 111 -> 104 us.
// r: the sums of columns col .. col + 31 of row `row`; columns from N on are not stored.
template <int EPI>
__device__ __forceinline__ void store_sums32(const uint32_t (&r)[32], void* __restrict__ y, int row, int col, int N,
                                             const GluParams& gp) {
    if (EPI == 0) {
        bf16* o = reinterpret_cast<bf16*>(y) + (size_t)row * N + col;
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            if (col + v * 8 >= N) break;
            uint4 pk;
            pk.x = pack_bf16(__uint_as_float(r[v * 8 + 0]), __uint_as_float(r[v * 8 + 1]));
            pk.y = pack_bf16(__uint_as_float(r[v * 8 + 2]), __uint_as_float(r[v * 8 + 3]));
            pk.z = pack_bf16(__uint_as_float(r[v * 8 + 4]), __uint_as_float(r[v * 8 + 5]));
            pk.w = pack_bf16(__uint_as_float(r[v * 8 + 6]), __uint_as_float(r[v * 8 + 7]));
            *reinterpret_cast<uint4*>(o + v * 8) = pk;
        }
    } else if (EPI == 1 || EPI == 3) {
        bf16* o = reinterpret_cast<bf16*>(y) + (size_t)row * (N >> 1) + (col >> 1);
        float res[16];
        if (EPI == 1) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const float g = __uint_as_float(r[(i >> 2) * 8 + (i & 3)]), u = __uint_as_float(r[(i >> 2) * 8 + 4 + (i & 3)]);
                res[i] = g / (1.0f + expf(-g)) * u;
            }
        } else {
            // One form for all 16, chosen once: with the choice inside `glu_gate` every gate was a chain of its own behind two
            // branches.
            float g[16], u[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                g[i] = __uint_as_float(r[(i >> 2) * 8 + (i & 3)]);
                u[i] = __uint_as_float(r[(i >> 2) * 8 + 4 + (i & 3)]);
            }
            if (gp.limit != INFINITY) {         // (min and max with an infinity change nothing but a NaN, which has to stay one)
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    g[i] = fminf(g[i], gp.limit);
                    u[i] = fminf(fmaxf(u[i], -gp.limit), gp.limit);
                }
            }
            if (gp.shift != 0.f) {
#pragma unroll
                for (int i = 0; i < 16; ++i) u[i] += gp.shift;
            }
            if (gp.slope == INFINITY) {
#pragma unroll
                for (int i = 0; i < 16; ++i) res[i] = fmaxf(g[i], 0.f) * u[i];
            } else if (gp.cubic != 0.f && gp.limit == INFINITY && gp.shift == 0.f) {
                // gelu's tanh form, whose own error is far above that of the fast exponential and division
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const float z = fmaf(gp.cubic * g[i] * g[i], g[i], g[i]);
                    res[i] = __fdividef(g[i], 1.0f + __expf(-gp.slope * z)) * u[i];
                }
            } else if (gp.cubic != 0.f) {
#pragma unroll
                for (int i = 0; i < 16; ++i) res[i] = g[i] / (1.0f + expf(-gp.slope * fmaf(gp.cubic * g[i] * g[i], g[i], g[i]))) * u[i];
            } else {
#pragma unroll
                for (int i = 0; i < 16; ++i) res[i] = g[i] / (1.0f + expf(-gp.slope * g[i])) * u[i];
            }
        }
#pragma unroll
        for (int v = 0; v < 2; ++v) {
            if (col + v * 16 >= N) break;
            uint4 pk;
            pk.x = pack_bf16(res[v * 8 + 0], res[v * 8 + 1]);
            pk.y = pack_bf16(res[v * 8 + 2], res[v * 8 + 3]);
            pk.z = pack_bf16(res[v * 8 + 4], res[v * 8 + 5]);
            pk.w = pack_bf16(res[v * 8 + 6], res[v * 8 + 7]);
            *reinterpret_cast<uint4*>(o + v * 8) = pk;
        }
    }
}

// The float32 rows of EPI 2: columns col .. col + 31 of rows row0 .. row0 + 31, a row's sums a lane, by a whole warp.  Stored as they
// lie, an instruction would write 16 bytes of 32 rows; turned through 4 KB of shared memory (rows in 16-byte pieces, their
// places swapped by the row, so that neither side meets in a bank) it writes the 128 bytes of 4 rows.
constexpr int TURN_BYTES = 32 * 32 * 4;           // a warp's
__device__ __forceinline__ void store_rows_turned(const uint32_t (&r)[32], float4* turn, float* __restrict__ y, int row0, int col, int M, int N, bool ok) {
    const int lane = threadIdx.x & 31;
    __syncwarp();
#pragma unroll
    for (int v = 0; v < 8; ++v)
        turn[lane * 8 + (v ^ (lane & 7))] = make_float4(__uint_as_float(r[4 * v]), __uint_as_float(r[4 * v + 1]), __uint_as_float(r[4 * v + 2]),
                                                        __uint_as_float(r[4 * v + 3]));
    __syncwarp();
    const int piece = lane & 7, at = col + piece * 4;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int lr = j * 4 + (lane >> 3);
        if (ok && row0 + lr < M && at < N) *reinterpret_cast<float4*>(y + (size_t)(row0 + lr) * N + at) = turn[lr * 8 + (piece ^ (lr & 7))];
    }
}

}  // namespace tc
