// 32-bit matrix product on the fifth-generation tensor cores: C[M, N] = A[M, K] * W[N, K]^T for float32 matrices, sent here from k of 2,048 on.
//
// A float32 number from 2^-110 up is the sum of three bf16 numbers (8 bits each of its 24): x = x1 + x2 + x3, |x2| <= 2^-8 |x|, |x3| <= 2^-17 |x|.  Six of the nine
// products of two such sums are formed; the other three come to 2^-24 of x w at the most (both just above a power of two) and 0.39 x 2^-26 root mean square.
// (So over one to four terms the result is 1.03 to 1.2 times as far off as a chain of FMAs, which rounds that seldom; from about eight on it is closer.)  Each
// product is exact in the tensor core's float32 accumulator, and what an accumulator loses is its own truncation (measured: 0.37 of 2^-24 of it for every 16
// of k).  So w1 x1 has an accumulator of its own and the five small products share another; both are read out and added in float32, rounded to nearest, every 256
// of k (a segment):
//     C = ((s0 + s1) + s2) + ..,   s = (w1 x1) + (w3 x1 + w2 x2 + w1 x3 + w2 x1 + w1 x2)
// Off float64 by 2.5e-7 of the result at K 2048 and 8192 (normal numbers), where one chain of K FMAs is 8e-7 and 1.6e-6.  The segments and the order in
// them are the same in both kernels below and for any number of rows, so a row's result does not depend on what else is in the batch.
// Below 2^-110 (2^-102 where subnormal operands count as zeros) the third part has bits under the smallest bf16.  So the largest magnitude of every row of A
// and of W is taken along, and an output that what is lost could reach, that is, one whose terms' magnitudes come to less than K (x_max + w_max + 8) 2^-100, is
// worked out again as a chain of FMAs from the float32 operands; so is one that is not finite (infinities and NaN, and numbers that round to infinity in 8 bits, come out as that chain gives them).
//
// W is the M side of the instruction (128 features a tile), split on the way: TMA brings 128 x 32 floats, warps turn a row of 32 into three
// planes of bf16 and put them into tensor memory as the A operand.  The rows of A are the N side, from shared memory in three planes.
//
// Every mbarrier wait is bounded by a fifth of a second of wall time; one that runs out sets an error word, lets every role run to its end
// without further waiting, and the CTA still frees its tensor memory.
// Role in the reference: `x.matmul(w.t())`, crates/model/src/layers.rs:82.
#include "tcgen05_utils.cuh"
#include <float.h>
#include <stddef.h>
#include <math.h>
#include <mutex>

namespace {
using namespace tc;

constexpr int FT = 128;                     // features a tile
constexpr int SEG = 256;                    // k of a segment
// k of a stage, and for it: stages of a segment, bytes of float32 weights, columns of tensor memory that their three planes take
constexpr int KS = 32, SEG_STAGES = SEG / KS, RAW_BYTES = FT * KS * 4, A_COLS = 3 * KS / 2;             // few rows
constexpr int KM = 64, SEG_STAGES_M = SEG / KM, RAW_BYTES_M = FT * KM * 4, A_COLS_M = 3 * KM / 2;       // many
constexpr int MAX_RINGS = 4, MAX_A = 4;     // stages of a ring in shared memory, and of the planes of weights in tensor memory

struct Ctrl {
    uint64_t raw_full[MAX_RINGS], raw_empty[MAX_RINGS], b_full[MAX_RINGS], b_empty[MAX_RINGS], a_full[MAX_A], a_empty[MAX_A], acc_full[2], acc_empty[2];
    uint32_t tmem_base;
    int abort;
    uint32_t most;                  // magnitudes, as bits of bf16: the largest of the CTA's operands (few rows: rows and weights; many: weights),
    uint16_t w_most[2][FT];         // of each row of weights, by the two sets of splitting warps,
    uint16_t x_most[32];            // and of each row of A (few rows)
};
static_assert(offsetof(Ctrl, w_most) % 4 == 0 && offsetof(Ctrl, x_most) % 4 == 0, "two magnitudes to a word");

struct SplitArgs {
    const float* A;
    const float* W;
    float* C;
    long long lda, ldw, ldc;
    int M, N, K;
    int bn;             // rows of A a tile
    int stages;         // of k in all
    int raw_ring;       // stages of the ring of float32 weights, and of A's planes (many rows)
    int rings;
    int m_tiles;
    int per;            // segments of a CTA of the cluster (few rows)
    int early;          // the weights may be read before the kernel before has finished
    float lost;         // K 2^-100
    const float* x_most;    // the largest magnitude of every row of A, by pieces of ROW_PIECE (many rows)
    int pieces;
};

// Two floats as three pairs of bf16 whose sum they are, low half first.
__device__ __forceinline__ void split2(float a, float b, uint32_t& p1, uint32_t& p2, uint32_t& p3) {
    p1 = pack_bf16(a, b);
    a -= __uint_as_float(p1 << 16);
    b -= __uint_as_float(p1 & 0xffff0000u);
    p2 = pack_bf16(a, b);
    a -= __uint_as_float(p2 << 16);
    b -= __uint_as_float(p2 & 0xffff0000u);
    p3 = pack_bf16(a, b);
}
// The larger magnitudes of two pairs of bf16, half by half, whatever their signs (a NaN counts as nothing); the larger one of a pair; its value.
__device__ __forceinline__ uint32_t larger2(uint32_t most, uint32_t p) {
    uint32_t d;
    asm("max.xorsign.abs.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(most), "r"(p));
    return d;
}
__device__ __forceinline__ uint32_t larger_half(uint32_t most) { return max(most & 0x7fffu, most >> 16 & 0x7fffu); }
__device__ __forceinline__ float magnitude(uint32_t bits) { return __uint_as_float(bits << 16); }
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]),
                 "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
__device__ __forceinline__ void tmem_ld16_nowait(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
        : "memory");
}
// Shared-memory matrix descriptor of a K-major tile whose rows are 32 k (64 bytes, 64-byte swizzle: layout type 4, 512 bytes between groups of 8 rows)
// or 64 k (128 bytes, 128-byte swizzle) wide.
template <int KT> __device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
    static_assert(KT == 32 || KT == 64, "stage");
    return ((uint64_t)(addr >> 4) & 0x3FFFull) | (1ull << 16) | ((uint64_t)(KT * 16 >> 4) << 32) | (1ull << 46) | ((KT == 32 ? 4ull : 2ull) << 61);
}

// A value that is the same in all lanes, in a way that the compiler sees: what descriptors are made from stays in uniform registers, which
// is where tcgen05.mma takes them.
template <typename T> __device__ __forceinline__ T uniform(T v) { return __shfl_sync(0xffffffffu, v, 0); }

// A stage's products (KT of k) over `n` rows of A: planes of the weights from tensor memory column `a`, of the rows from shared memory at `b`, planes
// `plane` bytes apart; sums of w1 x1 in columns `main`, of the others in `small`.
template <int KT> __device__ __forceinline__ void stage_products(uint32_t main, uint32_t small, uint32_t a, uint32_t b, uint32_t plane, int n, bool first) {
    const uint32_t idesc = idesc_bf16(FT, n);
    const uint64_t b1 = smem_desc<KT>(b), b2 = smem_desc<KT>(b + plane), b3 = smem_desc<KT>(b + 2 * plane);
    const uint32_t a1 = a, a2 = a + KT / 2, a3 = a + KT;
#pragma unroll
    for (int k = 0; k < KT / 16; ++k) {         // 8 columns, or 32 bytes of a swizzled row, further along k
        const uint32_t on = first && k == 0 ? 0u : 1u;
        umma_bf16_ts(small, a3 + k * 8, b1 + k * 2, idesc, on);
        umma_bf16_ts(small, a2 + k * 8, b2 + k * 2, idesc, 1u);
        umma_bf16_ts(small, a1 + k * 8, b3 + k * 2, idesc, 1u);
        umma_bf16_ts(small, a2 + k * 8, b1 + k * 2, idesc, 1u);
        umma_bf16_ts(small, a1 + k * 8, b2 + k * 2, idesc, 1u);
        umma_bf16_ts(main, a1 + k * 8, b1 + k * 2, idesc, on);
    }
}

// One row of KT float32 weights (boxes of 32: 128 bytes, 128-byte swizzle) into its three planes in tensor memory.
// (`most`: the largest magnitudes so far.)
template <int KT> __device__ __forceinline__ void split_weights(const unsigned char* raw, int row, uint32_t taddr, uint32_t& most) {
#pragma unroll
    for (int kk = 0; kk < KT / 16; ++kk) {
        const unsigned char* src = raw + kk / 2 * (FT * 32 * 4) + row * (32 * 4);
        uint32_t p1[8], p2[8], p3[8];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const float4 v = *reinterpret_cast<const float4*>(src + (((kk % 2 * 4 + c) ^ (row & 7)) << 4));
            split2(v.x, v.y, p1[2 * c], p2[2 * c], p3[2 * c]);
            split2(v.z, v.w, p1[2 * c + 1], p2[2 * c + 1], p3[2 * c + 1]);
            most = larger2(larger2(most, p1[2 * c]), p1[2 * c + 1]);
        }
        tmem_st8(taddr + kk * 8, p1);
        tmem_st8(taddr + KT / 2 + kk * 8, p2);
        tmem_st8(taddr + KT + kk * 8, p3);
    }
    tmem_st_wait();
}

// The magnitude of a row whose numbers are all zeros as bf16: zero, or the smallest one if some of them are not zero.
__device__ __noinline__ float magnitude_below(const float* __restrict__ row, int K) {
    uint32_t bits = 0;
    int k = 0;
    for (; k + 3 < K; k += 4) {
        const uint4 v = *reinterpret_cast<const uint4*>(row + k);
        bits |= v.x | v.y | v.z | v.w;
    }
    for (; k < K; ++k) bits |= __float_as_uint(row[k]);
    return bits << 1 ? magnitude(1) : 0.f;
}
// An output that is not finite, or so small that the parts' sums may have lost some of it, as a chain of FMAs (`x`, `w`: the largest magnitudes of
// the two rows, whatever else the tile holds).  One that came out small because its terms cancel has lost nothing beside its rounding and stays (of
// ordinary rows one in four million is exactly zero).
__device__ __noinline__ float chain(const float* __restrict__ a, const float* __restrict__ b, int K, float v, float x, float w, float lost) {
    const float least = lost * (x + w + 8.f);
    if (fabsf(v) <= FLT_MAX) {
        if (x == 0.f || w == 0.f || fabsf(v) >= least) return v;
        float terms[4] = {};
        int k = 0;
#pragma unroll 8
        for (; k + 3 < K; k += 4) {
            const float4 p = *reinterpret_cast<const float4*>(a + k), q = *reinterpret_cast<const float4*>(b + k);
            terms[0] = fmaf(fabsf(p.x), fabsf(q.x), terms[0]);
            terms[1] = fmaf(fabsf(p.y), fabsf(q.y), terms[1]);
            terms[2] = fmaf(fabsf(p.z), fabsf(q.z), terms[2]);
            terms[3] = fmaf(fabsf(p.w), fabsf(q.w), terms[3]);
        }
        for (; k < K; ++k) terms[0] = fmaf(fabsf(a[k]), fabsf(b[k]), terms[0]);
        if ((terms[0] + terms[1]) + (terms[2] + terms[3]) >= least) return v;
    }
    float acc = 0.f;
    for (int k = 0; k < K; ++k) acc = fmaf(a[k], b[k], acc);
    return acc;
}
// Whether an output is one that `chain` has to look at; `least`: what its rows' magnitudes come to at the most.
__device__ __forceinline__ bool doubtful(float v, float least) { return !(fabsf(v) <= FLT_MAX && fabsf(v) >= least); }

// The rows of A in three planes, planes[p][m][0 .. pitch), zeros beyond K, and the largest magnitude of each piece of a row.  A piece a warp, eight
// loads in flight a lane.
constexpr int ROW_PIECE = 1024;
__global__ __launch_bounds__(256) void split_rows_kernel(const float* __restrict__ A, long long lda, bf16* __restrict__ planes, float* __restrict__ most, int M, int K,
                                                         int pitch, int pieces) {
    pdl_wait_and_trigger();
    const size_t plane = (size_t)M * pitch, units = (size_t)M * pieces;
    const int lane = threadIdx.x & 31;
    for (size_t u = (size_t)blockIdx.x * 8 + (threadIdx.x >> 5); u < units; u += (size_t)gridDim.x * 8) {
        const size_t m = u / pieces;
        const int k0 = (int)(u % pieces) * ROW_PIECE + lane * 4;
        const float* src = A + m * lda;
        bf16* dst = planes + m * pitch;
        float4 v[ROW_PIECE / 128];
#pragma unroll
        for (int i = 0; i < ROW_PIECE / 128; ++i) {
            const int k = k0 + i * 128;
            v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (k + 3 < K) v[i] = *reinterpret_cast<const float4*>(src + k);
            else {
                if (k < K) v[i].x = src[k];
                if (k + 1 < K) v[i].y = src[k + 1];
                if (k + 2 < K) v[i].z = src[k + 2];
            }
        }
        uint32_t largest = 0, any = 0;
#pragma unroll
        for (int i = 0; i < ROW_PIECE / 128; ++i) {
            const int k = k0 + i * 128;
            uint2 p1, p2, p3;
            split2(v[i].x, v[i].y, p1.x, p2.x, p3.x);
            split2(v[i].z, v[i].w, p1.y, p2.y, p3.y);
            largest = larger2(larger2(largest, p1.x), p1.y);
            any |= __float_as_uint(v[i].x) | __float_as_uint(v[i].y) | __float_as_uint(v[i].z) | __float_as_uint(v[i].w);
            if (k < pitch) {
                *reinterpret_cast<uint2*>(dst + k) = p1;
                *reinterpret_cast<uint2*>(dst + plane + k) = p2;
                *reinterpret_cast<uint2*>(dst + 2 * plane + k) = p3;
            }
        }
        largest = __reduce_max_sync(0xffffffffu, max(larger_half(largest), any << 1 ? 1u : 0u));
        if (lane == 0) most[u] = magnitude(largest);
    }
}

// ------------------------------------------------------------------------------------------------
// Many rows.  700 rows, us here and in FFMA tiles: K 2048 N 16384 243 / 1139, N 3072 50 / 218, N 2048 38 / 218; K 8192 N 2048 130 / 858; 2,048 rows of K 2048 N 16384
// 646 / 2648 (213 TFLOP/s, six times that on the tensor cores: 1.3 PFLOP/s).  A stage takes the products' time (12 cycles a row) and about 1,100 cycles
// beside it, whatever the depth of the rings, so stages of 64 k are better than stages of 32 for tiles of few rows (48 rows 27 / 33 us, 200 39 / 50).
// A tile of 128 features x bn rows of A a CTA (bn up to 160), in two halves of the rows with accumulators, an issuing warp and four adding
// warps of their own: one warp alone spends more cycles between the bursts of two stages than the pipe has instructions queued.
// The rings have an even number of stages: a set meets the same ones every time, and so sees every phase of their barriers.
// Twenty warps, by role: 0-7 add the segments up and store, 8-15 split weights (two sets, taking turns at the stages), 16 and 17 ask for weights
// and for A's planes, 18 and 19 issue the products.
constexpr int MANY_THREADS = 640, MAX_BN = 160, HALF = MAX_BN / 2;
constexpr int MANY_RING_BYTES = 225 * 1024;         // both rings
constexpr int MANY_SMEM = 1024 + MANY_RING_BYTES + (int)sizeof(Ctrl);
static_assert(MANY_SMEM <= 227 * 1024, "shared memory");

__device__ __noinline__ float settle_many(const SplitArgs& p, int m, int n, float v, float w) {
    float x = 0.f;
    for (int i = 0; i < p.pieces; ++i) x = fmaxf(x, p.x_most[(size_t)m * p.pieces + i]);
    return chain(p.A + (size_t)m * p.lda, p.W + (size_t)n * p.ldw, p.K, v, x, w, p.lost);
}

__global__ __launch_bounds__(MANY_THREADS, 1) void f32_split_many_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a,
                                                                         const __grid_constant__ SplitArgs p) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* raw = base;
    unsigned char* planes = base + p.raw_ring * RAW_BYTES_M;
    Ctrl* ctrl = reinterpret_cast<Ctrl*>(base + MANY_RING_BYTES);
    const int warp = uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int f0 = (int)(blockIdx.x / p.m_tiles) * FT, m0 = (int)(blockIdx.x % p.m_tiles) * p.bn;
    const int n0 = (p.bn / 2 + 15) / 16 * 16, n1 = p.bn - n0;      // rows of the halves (the second has none where bn is 16)
    const uint32_t plane = (uint32_t)p.bn * (KM * 2), b_bytes = 3 * plane;
    const int a_ring = min(MAX_A, (512 - 4 * n0) / A_COLS_M) & ~1;

    if (threadIdx.x == 0) {
        ctrl->abort = 0;
        ctrl->most = 0;
        for (int i = 0; i < MAX_RINGS; ++i) {
            bar_init(&ctrl->raw_full[i], 1);
            bar_init(&ctrl->raw_empty[i], 4);
            bar_init(&ctrl->b_full[i], 1);
            bar_init(&ctrl->b_empty[i], n1 > 0 ? 2 : 1);
        }
        for (int i = 0; i < MAX_A; ++i) {
            bar_init(&ctrl->a_full[i], 4);
            bar_init(&ctrl->a_empty[i], n1 > 0 ? 2 : 1);
        }
        for (int i = 0; i < 2; ++i) {
            bar_init(&ctrl->acc_full[i], 1);
            bar_init(&ctrl->acc_empty[i], 4);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 18) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctrl->tmem_base)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = uniform(ctrl->tmem_base), a_base = tmem + 4 * n0;     // halves of [w1 x1 | the rest], n0 columns each; planes of weights

    if (warp >= 16) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
        if (warp == 16) {
            if (lane == 0) {
                if (!p.early) pdl_wait();
                for (int it = 0, s = 0, turn = 0; it < p.stages; ++it) {
                    if (turn > 0 && !bar_wait(&ctrl->raw_empty[s], (turn - 1) & 1, &ctrl->abort)) break;
                    bar_expect_tx(&ctrl->raw_full[s], RAW_BYTES_M);
                    tma_load_2d(raw + s * RAW_BYTES_M, &map_w, it * KM, f0, &ctrl->raw_full[s]);
                    tma_load_2d(raw + s * RAW_BYTES_M + RAW_BYTES_M / 2, &map_w, it * KM + 32, f0, &ctrl->raw_full[s]);
                    if (++s == p.raw_ring) { s = 0; ++turn; }
                }
            }
        } else if (warp == 17) {
            if (lane == 0) {
                pdl_wait();
                for (int it = 0, s = 0, turn = 0; it < p.stages; ++it) {
                    if (turn > 0 && !bar_wait(&ctrl->b_empty[s], (turn - 1) & 1, &ctrl->abort)) break;
                    bar_expect_tx(&ctrl->b_full[s], b_bytes);
                    tma_load_3d(planes + (size_t)s * b_bytes, &map_a, it * KM, m0, 0, &ctrl->b_full[s]);
                    if (++s == p.rings) { s = 0; ++turn; }
                }
            }
        } else if (warp == 18 || n1 > 0) {
            const int h = warp - 18, n = h ? n1 : n0;
            const uint32_t main = tmem + (uint32_t)(h * 2 * n0), rows = smem_u32(planes) + (uint32_t)(h * n0) * (KM * 2);
            int s = 0, a = 0;
            uint32_t a_turn = 0;
            for (int it = 0; it < p.stages; ++it) {
                const bool first = it % SEG_STAGES_M == 0, last = it % SEG_STAGES_M == SEG_STAGES_M - 1 || it == p.stages - 1;
                if (first && it > 0 && !bar_wait_warp(&ctrl->acc_empty[h], (it / SEG_STAGES_M - 1) & 1, &ctrl->abort)) break;
                if (!bar_wait_warp(&ctrl->a_full[a], a_turn, &ctrl->abort)) break;           // the rows' planes are there, too
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (elect_one()) {
                    stage_products<KM>(main, main + n0, a_base + (uint32_t)(a * A_COLS_M), rows + (uint32_t)s * b_bytes, plane, n, first);
                    umma_commit(&ctrl->a_empty[a]);
                    umma_commit(&ctrl->b_empty[s]);
                    if (last) umma_commit(&ctrl->acc_full[h]);
                }
                __syncwarp();
                if (++s == p.rings) s = 0;
                if (++a == a_ring) { a = 0; a_turn ^= 1; }
            }
        }
    } else if (warp >= 8) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
        const int set = (warp - 8) / 4, row = (warp & 3) * 32 + lane;
        const uint32_t taddr = a_base + ((uint32_t)((warp & 3) * 32) << 16);
        int s = set, a = set, b = set % p.rings;
        uint32_t turn = 0, a_turn = 0, b_turn = set / p.rings, most = 0;
        for (int it = set; it < p.stages; it += 2) {
            if (!bar_wait_warp(&ctrl->raw_full[s], turn & 1, &ctrl->abort)) break;
            if (a_turn > 0 && !bar_wait_warp(&ctrl->a_empty[a], (a_turn - 1) & 1, &ctrl->abort)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            split_weights<KM>(raw + s * RAW_BYTES_M, row, taddr + (uint32_t)(a * A_COLS_M), most);
            if (!bar_wait_warp(&ctrl->b_full[b], b_turn & 1, &ctrl->abort)) break;
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                bar_arrive(&ctrl->a_full[a]);
                bar_arrive(&ctrl->raw_empty[s]);
            }
            s += 2;
            if (s >= p.raw_ring) { s -= p.raw_ring; ++turn; }
            a += 2;
            if (a >= a_ring) { a -= a_ring; ++a_turn; }
            b += 2;
            if (b >= p.rings) { b -= p.rings; ++b_turn; }
        }
        most = larger_half(most);
        ctrl->w_most[set][row] = (uint16_t)most;
        most = __reduce_max_sync(0xffffffffu, most);
        if (lane == 0) atomicMax(&ctrl->most, most);
        asm volatile("bar.arrive 1, 512;" ::: "memory");
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 152;");
        const int h = warp >> 2, q = warp & 3, cols = h ? n1 : n0, segs = cols == 0 ? 0 : (p.stages + SEG_STAGES_M - 1) / SEG_STAGES_M;
        const uint32_t main = tmem + (uint32_t)(h * 2 * n0) + ((uint32_t)(q * 32) << 16);
        const int m1 = m0 + h * n0;
        float sum[HALF], x = 0.f;
#pragma unroll
        for (int c = 0; c < HALF; ++c) sum[c] = 0.f;
        pdl_wait();         // (C may still be read by the kernel before, too)
        for (int i = m1 * p.pieces + lane; i < min(m1 + cols, p.M) * p.pieces; i += 32) x = fmaxf(x, p.x_most[i]);
        x = warp_max(x);
        for (int seg = 0; seg < segs; ++seg) {
            if (!bar_wait_warp(&ctrl->acc_full[h], seg & 1, &ctrl->abort)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int c = 0; c < HALF / 16; ++c) {
                if (c * 16 < cols) {
                    uint32_t a[16], b[16];
                    tmem_ld16_nowait(main + c * 16, a);
                    tmem_ld16_nowait(main + n0 + c * 16, b);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; ++j) sum[c * 16 + j] += __uint_as_float(a[j]) + __uint_as_float(b[j]);
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) bar_arrive(&ctrl->acc_empty[h]);
        }
        const int n = f0 + q * 32 + lane;
        asm volatile("bar.sync 1, 512;" ::: "memory");        // the weights' magnitudes are there
        const float least = p.lost * (x + magnitude(ctrl->most) + 8.f);
        if (n < p.N && !ctrl->abort) {
            float w = magnitude(max(ctrl->w_most[0][q * 32 + lane], ctrl->w_most[1][q * 32 + lane]));
            if (w == 0.f) w = magnitude_below(p.W + (size_t)n * p.ldw, p.K);
#pragma unroll
            for (int c = 0; c < HALF; ++c)
                if (c < cols && m1 + c < p.M) {
                    const int m = m1 + c;
                    p.C[(size_t)m * p.ldc + n] = doubtful(sum[c], least) ? settle_many(p, m, n, sum[c], w) : sum[c];
                }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 18) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
    pdl_trigger();
}

// ------------------------------------------------------------------------------------------------
// Few rows (a decode step): bound by the memory's rate over W, and below it by a stage's way through the roles (raw weights, planes, products: about
// 900 cycles with one CTA on an SM, 600 a stage with two).  8 rows, us here and as chains of FMAs: K 2048 N 2048 9.7 / 11.1, N 3072 11.3 / 16, N 16384 32 / 44,
// N 32000 52 / 83 (5.0 TB/s); K 8192 N 2048 24 / 38.  A tile of 128 features a cluster, whose CTAs take whole segments of k and leave their
// sums in shared memory; the cluster then adds them up in the order of k, each CTA for a share of the features.  The rows of A are split
// where the weights are.  Fourteen warps: 0-3 read the accumulators, 4-11 split (two sets), 12 asks for weights and rows, 13 issues the products.
constexpr int FEW_THREADS = 448, FEW_RING = 4, FEW_A = 4;     // (a ring of an even number of stages, as above)

template <int BN> struct Few {
    static constexpr int ROWS_BYTES = BN * KS * 4, STAGE = RAW_BYTES + ROWS_BYTES, PLANES = 3 * BN * KS * 2, ROW = FT * 4;
    static constexpr int ACC = BN == 16 ? 2 : 1;                // accumulators: of two segments where there is room for them
    static_assert(ACC * 2 * BN + FEW_A * A_COLS <= 256, "two CTAs an SM share its tensor memory");
    static constexpr int smem(int rows) { return 1024 + FEW_RING * STAGE + FEW_A * PLANES + rows * ROW + (int)sizeof(Ctrl); }
};

// (the rows' magnitudes in the cluster's CTAs, which have a part of k each)
__device__ __noinline__ float settle_few(const SplitArgs& p, Ctrl* ctrl, int parts, int m, int f, int n, float v) {
    uint32_t x = 0, w = 0;
    auto take = [](uint16_t* at, int i, uint32_t part) { return __float_as_uint(ld_dsmem(reinterpret_cast<float*>(at + (i & ~1)), part)) >> (i & 1) * 16 & 0xffffu; };
    for (int part = 0; part < parts; ++part) {
        x = max(x, take(ctrl->x_most, m, (uint32_t)part));
        w = max(w, max(take(ctrl->w_most[0], f, (uint32_t)part), take(ctrl->w_most[1], f, (uint32_t)part)));
    }
    const float *a = p.A + (size_t)m * p.lda, *b = p.W + (size_t)n * p.ldw;
    return chain(a, b, p.K, v, x ? magnitude(x) : magnitude_below(a, p.K), w ? magnitude(w) : magnitude_below(b, p.K), p.lost);
}

template <int BN>
// (16 warps, to which 14 are rounded up, of two CTAs an SM have 64 registers a thread; 32 rows leave no room for a second one)
__global__ __launch_bounds__(BN == 16 ? 512 : FEW_THREADS, BN == 16 ? 2 : 1) void f32_split_few_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a,
                                                                       const __grid_constant__ SplitArgs p, int parts) {
    using F = Few<BN>;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* ring = base;                                             // weights, then rows
    unsigned char* planes = base + FEW_RING * F::STAGE;
    float* sums = reinterpret_cast<float*>(planes + FEW_A * F::PLANES);     // [segment of this CTA][row][feature]
    Ctrl* ctrl = reinterpret_cast<Ctrl*>(reinterpret_cast<unsigned char*>(sums) + (parts == 1 ? 1 : p.per) * p.M * F::ROW);
    const int warp = uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int f0 = (int)(blockIdx.x / parts) * FT, part = (int)(blockIdx.x % parts);
    const int segs = (p.stages + SEG_STAGES - 1) / SEG_STAGES;
    const int seg0 = min(part * p.per, segs), mine = min(segs - seg0, p.per);
    const int st0 = seg0 * SEG_STAGES, stages = max(0, min(p.stages, (seg0 + mine) * SEG_STAGES) - st0);

    if (threadIdx.x == 0) {
        ctrl->abort = 0;
        ctrl->most = 0;
        for (int i = 0; i < MAX_RINGS; ++i) {
            bar_init(&ctrl->raw_full[i], 1);
            bar_init(&ctrl->raw_empty[i], 8);
        }
        for (int i = 0; i < FEW_A; ++i) {
            bar_init(&ctrl->a_full[i], 8);
            bar_init(&ctrl->a_empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            bar_init(&ctrl->acc_full[i], 1);
            bar_init(&ctrl->acc_empty[i], 4);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 13) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctrl->tmem_base)), "r"(256) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = uniform(ctrl->tmem_base), a_base = tmem + F::ACC * 2 * BN;

    if (warp == 12) {
        if (lane == 0) {
            // weights that no kernel of a step writes are asked for before the wait; the rows after it
            if (!p.early) pdl_wait();
            const int early = min(stages, FEW_RING);
            for (int it = 0; it < early; ++it) {
                bar_expect_tx(&ctrl->raw_full[it], F::STAGE);
                tma_load_2d(ring + it * F::STAGE, &map_w, (st0 + it) * KS, f0, &ctrl->raw_full[it]);
            }
            pdl_wait();
            for (int it = 0; it < early; ++it) tma_load_2d(ring + it * F::STAGE + RAW_BYTES, &map_a, (st0 + it) * KS, 0, &ctrl->raw_full[it]);
            for (int it = early, s = 0, turn = 1; it < stages; ++it) {
                if (!bar_wait(&ctrl->raw_empty[s], (turn - 1) & 1, &ctrl->abort)) break;
                unsigned char* dst = ring + s * F::STAGE;
                bar_expect_tx(&ctrl->raw_full[s], F::STAGE);
                tma_load_2d(dst, &map_w, (st0 + it) * KS, f0, &ctrl->raw_full[s]);
                tma_load_2d(dst + RAW_BYTES, &map_a, (st0 + it) * KS, 0, &ctrl->raw_full[s]);
                if (++s == FEW_RING) { s = 0; ++turn; }
            }
            pdl_trigger();
        }
    } else if (warp == 13) {
        for (int it = 0; it < stages; ++it) {
            const int seg = it / SEG_STAGES, buf = seg % F::ACC, a = it % FEW_A;
            const bool first = it % SEG_STAGES == 0, last = it % SEG_STAGES == SEG_STAGES - 1 || it == stages - 1;
            if (first && seg >= F::ACC && !bar_wait_warp(&ctrl->acc_empty[buf], (seg / F::ACC - 1) & 1, &ctrl->abort)) break;
            if (!bar_wait_warp(&ctrl->a_full[a], (it / FEW_A) & 1, &ctrl->abort)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (elect_one()) {
                const uint32_t main = tmem + (uint32_t)(buf * 2 * BN);
                stage_products<KS>(main, main + BN, a_base + (uint32_t)(a * A_COLS), smem_u32(planes) + (uint32_t)(a * F::PLANES), BN * KS * 2, BN, first);
                umma_commit(&ctrl->a_empty[a]);
                if (last) umma_commit(&ctrl->acc_full[buf]);
            }
            __syncwarp();
        }
    } else if (warp >= 4) {
        const int set = (warp - 4) / 4, row = (warp & 3) * 32 + lane;
        const uint32_t taddr = a_base + ((uint32_t)((warp & 3) * 32) << 16);
        int s = set, turn = 0;
        uint32_t most = 0;
        for (int it = set; it < stages; it += 2) {
            const int a = it % FEW_A;
            if (!bar_wait_warp(&ctrl->raw_full[s], turn & 1, &ctrl->abort)) break;
            if (it >= FEW_A && !bar_wait_warp(&ctrl->a_empty[a], (it / FEW_A - 1) & 1, &ctrl->abort)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            split_weights<KS>(ring + s * F::STAGE, row, taddr + (uint32_t)(a * A_COLS), most);
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                bar_arrive(&ctrl->a_full[a]);
                bar_arrive(&ctrl->raw_empty[s]);
            }
            s += 2;
            if (s >= FEW_RING) { s -= FEW_RING; ++turn; }
        }
        most = larger_half(most);
        ctrl->w_most[set][row] = (uint16_t)most;
        most = __reduce_max_sync(0xffffffffu, most);
        if (lane == 0) atomicMax(&ctrl->most, most);
    } else {
        // the rows' planes, stage by stage, and behind each segment its sums
        const int f = threadIdx.x;
        auto take = [&](int seg) {
            const int buf = seg % F::ACC;
            if (!bar_wait_warp(&ctrl->acc_full[buf], (seg / F::ACC) & 1, &ctrl->abort)) return false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t main = tmem + (uint32_t)(buf * 2 * BN) + ((uint32_t)(warp * 32) << 16);
            float* dst = sums + (parts == 1 ? 0 : seg * p.M * FT) + f;
#pragma unroll
            for (int c = 0; c < BN / 16; ++c) {
                uint32_t a[16], b[16];
                tmem_ld16_nowait(main + c * 16, a);
                tmem_ld16_nowait(main + BN + c * 16, b);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    if (c * 16 + j >= p.M) break;
                    const float v = __uint_as_float(a[j]) + __uint_as_float(b[j]);
                    float* at = dst + (c * 16 + j) * FT;
                    *at = parts == 1 ? (seg == 0 ? 0.f : *at) + v : v;
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) bar_arrive(&ctrl->acc_empty[buf]);
            return true;
        };
        int s = 0, turn = 0, taken = 0;
        bool fine = true;
        uint32_t most[BN / 16] = {};
        for (int it = 0; it < stages; ++it) {
            const int a = it % FEW_A;
            // a segment's sums are due before the products that wait for their accumulator, and not before its last products are on their way
            if (it / SEG_STAGES >= taken + F::ACC && !(fine = take(taken++))) break;
            if (!(fine = bar_wait_warp(&ctrl->raw_full[s], turn & 1, &ctrl->abort))) break;
            if (it >= FEW_A && !(fine = bar_wait_warp(&ctrl->a_empty[a], (it / FEW_A - 1) & 1, &ctrl->abort))) break;
            const unsigned char* src = ring + s * F::STAGE + RAW_BYTES;
            unsigned char* dst = planes + a * F::PLANES;
#pragma unroll
            for (int i = 0; i < BN / 16; ++i) {         // four numbers of a row of A into 64-byte rows, 64-byte swizzle
                const int r = i * 16 + (f >> 3), c = f & 7;
                const float4 v = *reinterpret_cast<const float4*>(src + r * (KS * 4) + ((c ^ (r & 7)) << 4));
                uint2 p1, p2, p3;
                split2(v.x, v.y, p1.x, p2.x, p3.x);
                split2(v.z, v.w, p1.y, p2.y, p3.y);
                most[i] = larger2(larger2(most[i], p1.x), p1.y);
                unsigned char* d = dst + r * (KS * 2) + (((c >> 1) ^ ((r >> 1) & 3)) << 4) + (c & 1) * 8;
                *reinterpret_cast<uint2*>(d) = p1;
                *reinterpret_cast<uint2*>(d + BN * KS * 2) = p2;
                *reinterpret_cast<uint2*>(d + 2 * BN * KS * 2) = p3;
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                bar_arrive(&ctrl->a_full[a]);
                bar_arrive(&ctrl->raw_empty[s]);
            }
            if (++s == FEW_RING) { s = 0; ++turn; }
        }
#pragma unroll
        for (int i = 0; i < BN / 16; ++i) {             // (while the last products are on their way)
            uint32_t x = larger_half(most[i]);
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) x = max(x, __shfl_xor_sync(0xffffffffu, x, o));
            if ((f & 7) == 0) ctrl->x_most[i * 16 + (f >> 3)] = (uint16_t)x;
            x = __reduce_max_sync(0xffffffffu, x);
            if (lane == 0) atomicMax(&ctrl->most, x);
        }
        while (fine && taken < mine) fine = take(taken++);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 13) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256) : "memory");
    }
    pdl_wait();             // (C may still be read by the kernel before, whose end one thread alone has waited for)
    if (parts == 1) {
        const float least = p.lost * (2.f * magnitude(ctrl->most) + 8.f);
        for (int i = threadIdx.x; i < p.M * FT; i += FEW_THREADS) {
            const int m = i / FT, n = f0 + i % FT;
            if (n < p.N && !ctrl->abort) p.C[(size_t)m * p.ldc + n] = doubtful(sums[i], least) ? settle_few(p, ctrl, 1, m, i % FT, n, sums[i]) : sums[i];
        }
    } else {
        cluster_sync_all();
        const int share = (FT + parts - 1) / parts, lo = part * share, width = max(0, min(FT - lo, share));
        uint32_t most = lane < parts ? __float_as_uint(ld_dsmem(reinterpret_cast<float*>(&ctrl->most), (uint32_t)lane)) : 0u;      // (beside the sums, not before them)
        for (int i0 = warp * 32; i0 < p.M * width; i0 += FEW_THREADS) {
            const int i = min(i0 + lane, p.M * width - 1), m = i / width, f = lo + i % width;
            float v = 0.f;
            for (int s0 = 0; s0 < segs; s0 += 8) {
                float x[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int seg = min(s0 + j, segs - 1);
                    x[j] = ld_dsmem(sums + (seg % p.per) * p.M * FT + m * FT + f, (uint32_t)(seg / p.per));
                }
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    if (s0 + j < segs) v += x[j];
            }
            const float least = p.lost * (2.f * magnitude(__reduce_max_sync(0xffffffffu, most)) + 8.f);
            if (i0 + lane < p.M * width && f0 + f < p.N && !ctrl->abort)
                p.C[(size_t)m * p.ldc + f0 + f] = doubtful(v, least) ? settle_few(p, ctrl, parts, m, f, f0 + f, v) : v;
        }
        cluster_sync_all();         // nobody leaves while another CTA reads its sums
    }
    pdl_trigger();
}

// A float32 [rows, K] matrix with boxes of 32 k x box_rows rows, 128-byte swizzle.
bool map_f32(CUtensorMap* map, const float* ptr, int rows, int K, long long ld, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (fn == nullptr) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)ld * 4};
    const cuuint32_t box[2] = {(cuuint32_t)KS, (cuuint32_t)box_rows}, estr[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// The three planes of `rows` rows, pitch apart, with boxes of 64 k x box_rows rows x 3 planes, 128-byte swizzle.
bool map_planes(CUtensorMap* map, const bf16* ptr, int rows, int pitch, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (fn == nullptr) return false;
    const cuuint64_t dims[3] = {(cuuint64_t)pitch, (cuuint64_t)rows, 3}, strides[2] = {(cuuint64_t)pitch * 2, (cuuint64_t)pitch * rows * 2};
    const cuuint32_t box[3] = {(cuuint32_t)KM, (cuuint32_t)box_rows, 3}, estr[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<bf16*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int sm_count() {
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

constexpr int FEW_ROWS = 32, MAX_PARTS = 12, SMEM_MOST = 227 * 1024, SMEM_HALF = 112 * 1024, MAX_DEVICES = 64;     // (with half, two CTAs an SM)
int g_bn = 0, g_parts = 0;      // held fixed by a measurement (0: automatic)

// What is set for the kernels of few rows once a device, and the clusters of 1 .. MAX_PARTS CTAs that are resident at a time with one CTA an SM and with two.
// (The runtime counts one CTA an SM for a kernel that allocates tensor memory.  Of the places of two, clusters of three and more fill 95 %, of nine and more
// 85 %: with 148 SMs 48 clusters of 6 take two rounds and 32 of 8 one, 24 of 11 two and 24 of 10 one.)
struct FewPlan {
    std::once_flag once;
    cudaError_t error = cudaSuccess;
    int clusters[2][MAX_PARTS + 1] = {};
};
template <int BN> const FewPlan* few_plan() {
    static FewPlan plans[MAX_DEVICES];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev >= MAX_DEVICES) return nullptr;
    FewPlan& plan = plans[dev];
    std::call_once(plan.once, [&] {
        plan.error = cudaFuncSetAttribute(f32_split_few_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MOST);
        if (plan.error == cudaSuccess) plan.error = cudaFuncSetAttribute(f32_split_few_kernel<BN>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        for (int parts = 1; parts <= MAX_PARTS && plan.error == cudaSuccess; ++parts) {
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = parts;
            attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(parts);
            cfg.blockDim = dim3(FEW_THREADS);
            cfg.dynamicSmemBytes = SMEM_MOST;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            plan.error = cudaOccupancyMaxActiveClusters(&plan.clusters[0][parts], f32_split_few_kernel<BN>, &cfg);
            plan.clusters[1][parts] = 2 * sm_count() * (parts > 8 ? 85 : parts > 2 ? 95 : 100) / (100 * parts);
        }
    });
    return &plan;
}

// CTAs a tile, from what one takes, in ns: a segment 2,850 and 45 a row alone on its SM (with 32 rows a tile 3,500 and 35), 4,200 and 85 beside another, both
// more with the CTAs that share the memory, and 2,100 or, with others of its cluster, 3,200 beside its segments.  A cluster has to fit into a GPC, so fewer CTAs
// than there are places may already be too many for one round.  us with 1, 2, 4, 6 and 8 CTAs a tile, 8 rows: N 16384 K 2048 34, 30, 35, 45, 41; N 32000 51, 58,
// 65, 85, 77; N 3072 28, 17, 12, 14, 10; N 2048 K 8192 103, 56, 31, 27, 26, with 11 22; N 6144 K 4096 55, 34, 28, 35, 32.  32 rows: N 3072 K 3072 56, 34, 21, 33, 31.
template <int BN> int choose_parts(const FewPlan& plan, int tiles, int segs, int M) {
    int parts = 1;
    double least = -1;
    for (int c = 1; c <= MAX_PARTS && c <= segs; ++c) {
        const int per = (segs + c - 1) / c, bytes = Few<BN>::smem((c == 1 ? 1 : per) * M);
        if (bytes > SMEM_MOST || plan.clusters[0][c] <= 0) continue;
        const bool two = bytes <= SMEM_HALF && tiles > plan.clusters[0][c];
        const double rounds = (double)tiles / plan.clusters[two][c], ctas = (double)c * (rounds < 1 ? tiles : plan.clusters[two][c]);
        const double segment = two ? 4200 + 85 * M + 8 * ctas : BN == 16 ? 2850 + 45 * M + 8.5 * ctas : 3500 + 35 * M + 5 * ctas;
        const double t = (rounds <= 3 ? ceil(rounds) : rounds + (two ? 0.4 : 0.6)) * (per * segment + (c > 1 ? 3200 : 2100));
        if (least < 0 || t < least) { least = t; parts = c; }
    }
    return parts;
}

template <int BN> int launch_few(SplitArgs p, cudaStream_t stream) {
    using F = Few<BN>;
    const FewPlan* plan = few_plan<BN>();
    if (plan == nullptr) return RLIS_ERR_UNSUPPORTED;
    if (plan->error != cudaSuccess) return (int)plan->error;
    const int tiles = (p.N + FT - 1) / FT, segs = (p.stages + SEG_STAGES - 1) / SEG_STAGES;
    int parts = choose_parts<BN>(*plan, tiles, segs, p.M);
    if (g_parts > 0 && g_parts <= segs && F::smem((g_parts == 1 ? 1 : (segs + g_parts - 1) / g_parts) * p.M) <= SMEM_MOST) parts = g_parts;
    p.per = (segs + parts - 1) / parts;
    CUtensorMap map_w, map_a;
    if (!map_f32(&map_w, p.W, p.N, p.K, p.ldw, FT) || !map_f32(&map_a, p.A, p.M, p.K, p.lda, BN)) return RLIS_ERR_UNSUPPORTED;
    const int smem = F::smem((parts == 1 ? 1 : p.per) * p.M);
    rlis_launch_cluster(f32_split_few_kernel<BN>, dim3((unsigned)(tiles * parts)), dim3(FEW_THREADS), (size_t)smem, stream, dim3((unsigned)parts, 1, 1), map_w, map_a, p, parts);
    return RLIS_LAUNCH_CHECK();
}

// Rows of A a tile: what takes the SMs least time.  Measured on 700 rows, in cycles a stage: 16 rows 1,300, 64 1,680, 96 2,160, 128 2,640, 160 3,050;
// a tile takes about 6,000 cycles beside its stages.
int choose_bn(int M, int N, int stages, int sms) {
    if (g_bn > 0) return g_bn;
    const long long f_tiles = (N + FT - 1) / FT;
    int best = 16;
    double least = -1;
    for (int bn = 16; bn <= MAX_BN; bn += 16) {
        const long long waves = (f_tiles * ((M + bn - 1) / bn) + sms - 1) / sms;
        const double t = (double)waves * (stages * (1070 + 12.2 * bn) + 6000);
        if (least < 0 || t < least) { least = t; best = bn; }
    }
    return best;
}
}  // namespace

extern "C" int rlis_gemm_f32_split_few_rows(void) { return FEW_ROWS; }
extern "C" void rlis_gemm_f32_split_set_rows(int n) { g_bn = n >= 16 && n <= MAX_BN && n % 16 == 0 ? n : 0; }
extern "C" void rlis_gemm_f32_split_set_parts(int n) { g_parts = n >= 0 && n <= MAX_PARTS ? n : 0; }

// Bytes of scratch a row (0: too long a row): its three planes and the magnitudes of its pieces.
extern "C" int rlis_gemm_f32_split_row_bytes(int K) { return K <= 0 || K > (1 << 28) ? 0 : 6 * ((K + 7) / 8 * 8) + 4 * ((K + ROW_PIECE - 1) / ROW_PIECE); }

// C[M, N] = A[M, K] W[N, K]^T, rows lda, ldw, ldc floats apart; A, W, lda and ldw on 16-byte boundaries, K >= 1.  More than
// rlis_gemm_f32_split_few_rows() rows: `planes` is scratch of M times rlis_gemm_f32_split_row_bytes(K) bytes on a 16-byte boundary.  `early`: no kernel
// that is still running writes W, so that its first tiles may be asked for before those before in the stream have finished.
extern "C" int rlis_gemm_f32_split(const float* A, long long lda, const float* W, long long ldw, float* C, long long ldc, int M, int N, int K, void* planes,
                                   int early, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || lda % 4 || ldw % 4 || ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W)) & 15)) return RLIS_ERR_UNSUPPORTED;
    SplitArgs p = {A, W, C, lda, ldw, ldc, M, N, K, 0, (K + KS - 1) / KS, 0, 0, 1, 0, early, K * 0x1p-100f, nullptr, (K + ROW_PIECE - 1) / ROW_PIECE};
    if (M <= 16) return launch_few<16>(p, stream);
    if (M <= FEW_ROWS) return launch_few<32>(p, stream);
    if (planes == nullptr || (reinterpret_cast<uintptr_t>(planes) & 15)) return RLIS_ERR_UNSUPPORTED;
    const int sms = sm_count(), pitch = (K + 7) / 8 * 8;
    float* most = reinterpret_cast<float*>(reinterpret_cast<bf16*>(planes) + (size_t)3 * M * pitch);
    const long long blocks = ((long long)M * p.pieces + 7) / 8;
    rlis_launch(split_rows_kernel, dim3((unsigned)(blocks < 8LL * sms ? blocks : 8LL * sms)), dim3(256), 0, stream, A, lda, reinterpret_cast<bf16*>(planes), most, M, K,
                pitch, p.pieces);
    int rc = RLIS_LAUNCH_CHECK();
    if (rc != 0) return rc;
    p.x_most = most;
    p.bn = choose_bn(M, N, (K + KM - 1) / KM, sms);
    p.m_tiles = (M + p.bn - 1) / p.bn;
    const int b_bytes = 3 * p.bn * KM * 2;
    p.stages = (K + KM - 1) / KM;
    p.rings = p.bn > 64 ? 2 : 4;
    p.raw_ring = p.rings * b_bytes + 4 * RAW_BYTES_M <= MANY_RING_BYTES ? 4 : 2;
    CUtensorMap map_w, map_a;
    if (!map_f32(&map_w, W, N, K, ldw, FT) || !map_planes(&map_a, reinterpret_cast<const bf16*>(planes), M, pitch, p.bn)) return RLIS_ERR_UNSUPPORTED;
    static std::atomic<unsigned long long> done{0};
    const cudaError_t e = rlis_allow_smem(f32_split_many_kernel, MANY_SMEM, done);
    if (e != cudaSuccess) return (int)e;
    const long long tiles = (long long)((N + FT - 1) / FT) * p.m_tiles;
    rlis_launch(f32_split_many_kernel, dim3((unsigned)tiles), dim3(MANY_THREADS), (size_t)MANY_SMEM, stream, map_w, map_a, p);
    return RLIS_LAUNCH_CHECK();
}

extern "C" int rlis_gemm_f32_split_error(void) { return tc::read_error_word(); }
extern "C" int* rlis_gemm_f32_split_error_addr(void) { return tc::error_word_addr(); }
