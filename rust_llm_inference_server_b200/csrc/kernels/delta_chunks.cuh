// The gated delta rule with one decay a head over prompts, 64 tokens at a time (heads of 128 x 128).  The notation is that of conv_recurrence.cuh: with
// L_t the sum of ln g over the chunk's tokens up to t, S0 the state before the chunk, A[t][i] = beta_t e^{L_t - L_i} k_t . k_i (i < t) and
// T = (I + A)^-1,
//
//   u = T (beta v) - W S0,  W = T (beta e^L k);   o_t = e^{L_t} S0^T q_t + sum_{i <= t} e^{L_t - L_i} (q_t . k_i) u_i;   S = e^{L_end} S0 + sum_t e^{L_end - L_t} k_t u_t^T
//
// which is the recurrence written out (the compact WY form of products of Householder-like factors).  Only u and S go from chunk to chunk, two products of 64 x 128 a column block; everything else is done for all
// chunks at once, before and after:
//   delta_chunk_prepare: (chunk, head)  T, T (beta v), W, the decayed q . k, the powers of the decay
//   delta_chunk_walk:    (request, head, 16 columns)  the chunks in order: u, and the state before every chunk
//   delta_chunk_outputs: (chunk, head, 64 columns)  o
// Everything is float32 (FFMA, two at a time), sums in blocks of 8, L as the sum of two floats.  409 and 1,092 tokens, 16 heads: 77, 119 and 48 us, where the
// kernels for 16 tokens take 356 (a chain of 69 chunks of shuffles and barriers); off 64 bits by 1.5e-7 of the outputs (2.4e-7 there, 7.6e-7 with L in one
// float).  No pipe is near its limit: the FMA pipe, shared memory and the issue slots are busy 48, 44 and 44 % of the time in the first kernel, 40, 39 and 34 in the walk, 42,
// 36 and 31 in the last.  What bounds them is the latency of reads and barriers with 16, 16 and 8 warps an SM (three 16-byte reads feed 32 FMAs a thread) and, with
// few heads, the chain.
#pragma once
#include "chunk_products.cuh"

namespace convrec {
namespace wide {
using namespace chunkprod;
constexpr int D = 128, LDR = D + 4, VT = 64, WC = 16;       // heads; rows of 128; columns of v a CTA of the outputs, and of the walk
constexpr int PREPARE_THREADS = 256, WALK_THREADS = 256, OUTPUT_THREADS = 128;
// The least ln g that is summed: its power is 0 like that of anything below, and the differences of the sums over tokens behind it keep their bits (ln g comes
// as low as -1e30, and from about 1e16 on the rounding of a sum of two such, left in the second float, leaves nothing there of ordinary ones).
constexpr float LEAST = -1024.f;

// Scratch of a (chunk, head), in floats: decayed q . k [key][query], W turned [entry][token], u [token][dv], the state before the
// chunk [entry][dv], e^{L_end - L} and e^L.
struct Unit {
    float *p, *w, *u, *s, *tail, *grow;
    __device__ __forceinline__ Unit(float* base, size_t unit, int dv)
        : p(base + unit * size(dv)), w(p + CHUNK * CHUNK), u(w + D * CHUNK), s(u + CHUNK * dv), tail(s + D * dv), grow(tail + CHUNK) {}
    __host__ __device__ static constexpr size_t size(int dv) { return (size_t)CHUNK * CHUNK + D * CHUNK + (size_t)(CHUNK + D) * dv + 2 * CHUNK; }
};
// Chunk c of the step: its first token's row and its tokens (none: there is no such chunk).
__device__ __forceinline__ int2 chunk_rows(const Seqs& s, int n_seqs, int c) {
    for (int b = 0; b < n_seqs; ++b) {
        const int row = s.cu_seqlens[b], n = s.cu_seqlens[b + 1] - row, chunks = (n + CHUNK - 1) / CHUNK;
        if (c < chunks) return make_int2(row + c * CHUNK, min(CHUNK, n - c * CHUNK));
        c -= chunks;
    }
    return make_int2(0, 0);
}
// Rows of 128 floats `ld` apart, turned: [entry][64 rows + 4]; rows from n on become zeros.
template <int THREADS> __device__ __forceinline__ void stage_turned(float* dst, const float* x, size_t ld, int n) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll 4
    for (int i = warp; i < CHUNK / 8 * (D / 16); i += THREADS / 32) {
        const int r = i % (CHUNK / 8) * 8 + lane % 8, c = (i / (CHUNK / 8) * 4 + lane / 8) * 4;
        const float4 v = r < n ? load_quad(x + r * ld + c) : make_float4(0.f, 0.f, 0.f, 0.f);
        dst[c * LDT + r] = v.x; dst[(c + 1) * LDT + r] = v.y; dst[(c + 2) * LDT + r] = v.z; dst[(c + 3) * LDT + r] = v.w;
    }
}

// The sum of two numbers kept as sums of two floats (what a float sum leaves out, exactly, beside it: Knuth's two-sum).
__device__ __forceinline__ float2 two_sum(float2 a, float2 b) {
    const float s = __fadd_rn(a.x, b.x), t = __fsub_rn(s, a.x);
    return make_float2(s, __fadd_rn(__fadd_rn(__fsub_rn(a.x, __fsub_rn(s, t)), __fsub_rn(b.x, t)), __fadd_rn(a.y, b.y)));
}
// e^(hi + lo) for a lo of at most half a unit of hi; e^(a - b)
__device__ __forceinline__ float exp_of(float2 v) {
    const float e = expf(v.x);
    return fmaf(e, v.y, e);
}
__device__ __forceinline__ float exp_between(float2 a, float2 b) { return expf((a.x - b.x) + (a.y - b.y)); }

template <int>
__global__ __launch_bounds__(PREPARE_THREADS, 2) void delta_chunk_prepare(const float* __restrict__ act, float* __restrict__ scratch, Seqs sq, int n_seqs, Shape z) {
    extern __shared__ __align__(16) float smem[];
    float* kt = smem;                       // keys turned, then beta v by rows
    float* qt = kt + D * LDT;               // queries turned, then beta e^L k by rows
    float* am = qt + D * LDT;               // [token][token + 4] A
    float* tt = am + CHUNK * LDT;           // [column][row + 4] T
    float* xs = tt + CHUNK * LDT;           // three blocks of 16 x 17
    __shared__ __align__(16) float2 ls[CHUNK];            // L as the sum of two floats: a difference of two is as exact as its size allows
    __shared__ __align__(8) float bs[CHUNK];
    pdl_wait();
    const int2 rows = chunk_rows(sq, n_seqs, blockIdx.x);
    if (rows.y > 0) {
        const int h = blockIdx.y, hq = h / (z.nh / z.n_qk), n = rows.y, C = z.channels(), dv = z.dv;
        const size_t AW = act_width<HEAD_DECAY>(z);
        const float* x = act + rows.x * AW;
        const Unit out(scratch, (size_t)blockIdx.x * z.nh + h, dv);
        if (threadIdx.x < 32) {             // two tokens a lane
            const int a = 2 * threadIdx.x;
            const float g0 = a < n ? fmaxf(x[a * AW + C + z.nh + h], LEAST) : 0.f, g1 = a + 1 < n ? fmaxf(x[(a + 1) * AW + C + z.nh + h], LEAST) : 0.f;
            const float b0 = a < n ? x[a * AW + C + h] : 0.f, b1 = a + 1 < n ? x[(a + 1) * AW + C + h] : 0.f;
            float2 L = two_sum(make_float2(g0, 0.f), make_float2(g1, 0.f));
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float2 up = make_float2(__shfl_up_sync(0xffffffffu, L.x, o), __shfl_up_sync(0xffffffffu, L.y, o));
                if ((int)threadIdx.x >= o) L = two_sum(L, up);
            }
            const float2 before = make_float2(__shfl_up_sync(0xffffffffu, L.x, 1), __shfl_up_sync(0xffffffffu, L.y, 1));
            const float2 end = make_float2(__shfl_sync(0xffffffffu, L.x, 31), __shfl_sync(0xffffffffu, L.y, 31));
            const float2 L0 = threadIdx.x > 0 ? two_sum(before, make_float2(g0, 0.f)) : make_float2(g0, 0.f);
            *reinterpret_cast<float4*>(ls + a) = make_float4(L0.x, L0.y, L.x, L.y);
            *reinterpret_cast<float2*>(bs + a) = make_float2(b0, b1);
            *reinterpret_cast<float2*>(out.grow + a) = make_float2(exp_of(L0), exp_of(L));
            *reinterpret_cast<float2*>(out.tail + a) = make_float2(exp_between(end, L0), exp_between(end, L));
        }
        stage_turned<PREPARE_THREADS>(kt, x + z.k_at + hq * D, AW, n);
        stage_turned<PREPARE_THREADS>(qt, x + z.q_at + hq * D, AW, n);
        __syncthreads();
        const int t = threadIdx.x & 127, group = threadIdx.x >> 7, ty = thread_row(t), tx = thread_col(t);
        Tile<4> acc;
        acc.clear();
        product<4, 8>(acc, group ? qt : kt, LDT, kt, LDT, D, ty, tx);
#pragma unroll
        for (int i0 = 0; i0 < 8; i0 += 4) {
            const int r = i0 * 8 + ty * 4;
            float v[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float b = group ? 1.0f : bs[r + i];
                const float2 L = ls[r + i];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int c = tx * 4 + j;
                    if (r < tx * 4) v[i][j] = 0.f;
                    else v[i][j] = (group ? r + i >= c : r + i > c) ? b * exp_between(L, ls[c]) * acc.at(i0 + i, j) : 0.f;
                }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (group) *reinterpret_cast<float4*>(out.p + (tx * 4 + j) * CHUNK + r) = make_float4(v[0][j], v[1][j], v[2][j], v[3][j]);
                else *reinterpret_cast<float4*>(am + (r + j) * LDT + tx * 4) = make_float4(v[j][0], v[j][1], v[j][2], v[j][3]);
            }
        }
        for (int i = threadIdx.x; i < CHUNK * LDT; i += PREPARE_THREADS) tt[i] = 0.f;
        __syncthreads();
        // T by blocks of 16: those on the diagonal column by column, the others a distance from it at a time.  (Sums stop where a row's tokens
        // end: what is not finite in a later token reaches no earlier one.)
        if (threadIdx.x < CHUNK) {
            const int b0 = threadIdx.x & ~15, j = threadIdx.x & 15;
            float col[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                float v = i == j ? 1.f : 0.f;
#pragma unroll
                for (int m = 0; m < i; ++m)
                    if (m >= j) v = fmaf(-am[(b0 + i) * LDT + b0 + m], col[m], v);
                col[i] = v;
                if (i >= j) tt[(b0 + j) * LDT + b0 + i] = v;
            }
        }
        __syncthreads();
        const int bi = threadIdx.x >> 4, bj = threadIdx.x & 15;
#pragma unroll
        for (int dist = 1; dist < 4; ++dist) {
            for (int r = dist; r < 4; ++r) {
                const int c = r - dist;
                const float *a = am + (r * 16 + bi) * LDT, *e = tt + (c * 16 + bj) * LDT;
                float v[4] = {};
                for (int p = c * 16; p < r * 16; p += 16)
#pragma unroll
                    for (int q = 0; q < 16; q += 4) {
                        const float4 x4 = load_quad(a + p + q), y4 = load_quad(e + p + q);
                        v[0] = fmaf(x4.x, y4.x, v[0]); v[1] = fmaf(x4.y, y4.y, v[1]); v[2] = fmaf(x4.z, y4.z, v[2]); v[3] = fmaf(x4.w, y4.w, v[3]);
                    }
                xs[(c * 16 + bi) * 17 + bj] = (v[0] + v[1]) + (v[2] + v[3]);
            }
            __syncthreads();
            for (int r = dist; r < 4; ++r) {
                const int c = r - dist;
                float v[4] = {};
#pragma unroll
                for (int p = 0; p < 16; ++p)
                    if (p <= bi) v[p & 3] = fmaf(tt[(r * 16 + p) * LDT + r * 16 + bi], xs[(c * 16 + p) * 17 + bj], v[p & 3]);
                tt[(c * 16 + bj) * LDT + r * 16 + bi] = -((v[0] + v[1]) + (v[2] + v[3]));
            }
            __syncthreads();
        }
        // T (beta v) a block of 128 columns at a time, and W
        for (int v0 = 0; v0 < dv; v0 += D) {
            bool met = false;
            auto put = [&](float* to, float4 v, float f) {
                v = make_float4(f * v.x, f * v.y, f * v.z, f * v.w);
                met |= !(fabsf(v.x) < INFINITY && fabsf(v.y) < INFINITY && fabsf(v.z) < INFINITY && fabsf(v.w) < INFINITY);
                *reinterpret_cast<float4*>(to) = v;
            };
#pragma unroll 4
            for (int i = threadIdx.x; i < CHUNK * D / 4; i += PREPARE_THREADS) {
                const int r = i / (D / 4), c = i % (D / 4) * 4;
                const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
                put(kt + r * LDR + c, r < n && v0 + c < dv ? load_quad(x + r * AW + z.v_at + h * dv + v0 + c) : none, bs[r]);
                if (v0 == 0) put(qt + r * LDR + c, r < n ? load_quad(x + r * AW + z.k_at + hq * D + c) : none, bs[r] * exp_of(ls[r]));
            }
            const bool spoilt = __syncthreads_or(met);
            if (group == 0 || v0 == 0) {
                const float* src = group ? qt : kt;
#pragma unroll 1
                for (int half = 0; half < 2; ++half) {
                    const int c0 = half * 64 + tx * 4;
                    if (group == 0 && v0 + half * 64 >= dv) break;
                    acc.clear();
                    if (!spoilt) product<4, 8>(acc, tt, LDT, src + half * 64, LDR, (n + 7) & ~7, ty, tx);
#pragma unroll
                    for (int i0 = 0; i0 < 8; i0 += 4) {
                        const int r = i0 * 8 + ty * 4;
                        float v[4][4];
#pragma unroll
                        for (int i = 0; i < 4; ++i)
#pragma unroll
                            for (int j = 0; j < 4; ++j) v[i][j] = acc.at(i0 + i, j);
                        if (spoilt) {       // a zero times what is not finite would reach tokens that came before it; the same sums without those
#pragma unroll
                            for (int i = 0; i < 4; ++i)
#pragma unroll
                                for (int j = 0; j < 4; ++j) {
                                    v[i][j] = 0.f;
#pragma unroll 1
                                    for (int k0 = 0; k0 <= r + i; k0 += 8) {
                                        float part = 0.f;
#pragma unroll 1
                                        for (int k = k0; k < k0 + 8 && k <= r + i; ++k) part = fmaf(tt[k * LDT + r + i], src[k * LDR + c0 + j], part);
                                        v[i][j] += part;
                                    }
                                }
                        }
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            if (group) *reinterpret_cast<float4*>(out.w + (c0 + j) * CHUNK + r) = make_float4(v[0][j], v[1][j], v[2][j], v[3][j]);
                            else *reinterpret_cast<float4*>(out.u + (size_t)(r + j) * dv + v0 + c0) = make_float4(v[j][0], v[j][1], v[j][2], v[j][3]);
                        }
                    }
                }
            }
            __syncthreads();
        }
    }
    pdl_trigger();
}

// Eight warps.  Both products are bound by reads of shared memory, so a thread has 8 x 4 outputs (three 16-byte reads for 32 FMAs) and the warps share out
// the terms instead: u: 16 entries a warp; the state: 16 tokens two warps.  What a share comes to is left where its operand was, and added up by all threads.
// W arrives (16-byte asynchronous copies) while the state takes the chunk before, the keys while u is formed.
// (A chunk with a CTA alone on its SM and with two: 9,100 and 15,000 cycles with 4 x 2 outputs a thread.)
template <typename T>
__global__ __launch_bounds__(WALK_THREADS, 2) void delta_chunk_walk(const float* __restrict__ act, float* __restrict__ scratch, float* __restrict__ state,
                                                                    long long state_stride, long long tail_off, const T* __restrict__ x_in, long long stride,
                                                                    Seqs sq, Shape z) {
    constexpr int LDC = WC + 4, SHARE = 16;
    static_assert(SHARE * WALK_THREADS / 32 == D && CHUNK * WC <= SHARE * LDT && D * WC <= SHARE * LDR && CHUNK / SHARE * 64 == WALK_THREADS, "shares");
    extern __shared__ __align__(16) float smem[];
    float* wt = smem;                       // [entry][token + 4]
    float* ks = wt + D * LDT;               // [token][entry + 4]
    float* st = ks + CHUNK * LDR;           // [entry][column + 4] the state
    float* us = st + D * LDC;               // [token][column + 4] u, decayed to the chunk's end
    pdl_wait();
    const int b = blockIdx.x, h = blockIdx.y, c0 = blockIdx.z * WC, hq = h / (z.nh / z.n_qk), dv = z.dv;
    const int row0 = sq.cu_seqlens[b], n = sq.cu_seqlens[b + 1] - row0;
    if (n > 0) {
        const bool fresh = sq.ctx_lens[b] - n == 0;
        float* slot = state + (size_t)sq.state_slots[b] * state_stride;
        if (z.taps > 1)
            move_tail<T, WALK_THREADS>(slot + tail_off, x_in, stride, row0, n, z.channels(), z.taps, fresh, h * gridDim.z + blockIdx.z, z.nh * gridDim.z);
        int before = 0;
        for (int o = 0; o < b; ++o) before += (sq.cu_seqlens[o + 1] - sq.cu_seqlens[o] + CHUNK - 1) / CHUNK;
        const size_t AW = act_width<HEAD_DECAY>(z);
        const float* keys = act + row0 * AW + z.k_at + hq * D;
        const int chunks = (n + CHUNK - 1) / CHUNK, tid = threadIdx.x;
        auto unit = [&](int c) { return Unit(scratch, (size_t)(before + c) * z.nh + h, dv); };
        auto ask_w = [&](int c) {
            if (c < chunks) {
                const float* w = unit(c).w + tid * 4;
                float* dst = wt + tid / (CHUNK / 4) * LDT + tid % (CHUNK / 4) * 4;
                constexpr int step = WALK_THREADS / (CHUNK / 4);
#pragma unroll
                for (int i = 0; i < D / step; ++i) cp_async16(dst + i * step * LDT, w + i * WALK_THREADS * 4, true);
            }
            cp_async_commit();
        };
        auto ask_k = [&](int c) {
            if (c < chunks) {
                const int r = tid / (D / 4), e = tid % (D / 4) * 4;
                const float* k = keys + e;
                float* dst = ks + r * LDR + e;
                constexpr int step = WALK_THREADS / (D / 4);
#pragma unroll
                for (int i = 0; i < CHUNK / step; ++i) {
                    const int row = c * CHUNK + r + i * step;
                    cp_async16(dst + i * step * LDR, k + (size_t)min(row, n - 1) * AW, row < n);
                }
            }
            cp_async_commit();
        };
        ask_w(0);
        ask_k(0);
        float* S = slot + ((size_t)h * dv + c0) * D;
        for (int i = tid; i < WC * D / 4; i += WALK_THREADS) {
            const int c = i / (D / 4), e = i % (D / 4) * 4;
            const float4 v = fresh ? make_float4(0.f, 0.f, 0.f, 0.f) : load_quad(S + c * D + e);
            st[e * LDC + c] = v.x; st[(e + 1) * LDC + c] = v.y; st[(e + 2) * LDC + c] = v.z; st[(e + 3) * LDC + c] = v.w;
        }
        const int lane = tid & 31, warp = tid >> 5, share = tid >> 6;
        const int uy = lane >> 2, sy = (warp & 1) * 8 + (lane >> 2), x = lane & 3;    // rows 4 y + {0..3} and those 32 (64) on, columns 4 x + {0..3}
        // place of four columns of a row among the sums of a share (rows of 16, shuffled so that a warp's writes spread over the banks)
        auto at = [](int row, int quad) { return row * WC + ((quad ^ (row >> 2)) & 3) * 4; };
        for (int c = 0; c < chunks; ++c) {
            const Unit m = unit(c);
            const int ut = tid >> 2;                            // this thread's token and columns of u
            float4 u = load_quad(m.u + (size_t)ut * dv + c0 + x * 4);
            const float f = m.tail[ut], whole = m.grow[CHUNK - 1];
            cp_async_wait<1>();
            __syncthreads();                // W and the state are there
#pragma unroll
            for (int i = 0; i < D * WC / 4 / WALK_THREADS; ++i) {
                const int e = (tid + i * WALK_THREADS) / (WC / 4), q = (tid + i * WALK_THREADS) % (WC / 4) * 4;
                *reinterpret_cast<float4*>(m.s + (size_t)e * dv + c0 + q) = *reinterpret_cast<const float4*>(st + e * LDC + q);
            }
            {
                Tile<4> acc;
                acc.clear();
                float* mine = wt + warp * SHARE * LDT;
                rows_product<32, 8>(acc, mine + uy * 4, LDT, st + warp * SHARE * LDC + x * 4, LDC, SHARE);
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    *reinterpret_cast<float4*>(mine + at(i / 4 * 32 + uy * 4 + i % 4, x)) = make_float4(acc.at(i, 0), acc.at(i, 1), acc.at(i, 2), acc.at(i, 3));
            }
            __syncthreads();
            {
                float4 s = *reinterpret_cast<const float4*>(wt + at(ut, x));
#pragma unroll
                for (int w = 1; w < D / SHARE; ++w) {
                    const float4 o = *reinterpret_cast<const float4*>(wt + w * SHARE * LDT + at(ut, x));
                    s.x += o.x; s.y += o.y; s.z += o.z; s.w += o.w;
                }
                u = make_float4(u.x - s.x, u.y - s.y, u.z - s.z, u.w - s.w);
                *reinterpret_cast<float4*>(m.u + (size_t)ut * dv + c0 + x * 4) = u;
                *reinterpret_cast<float4*>(us + ut * LDC + x * 4) = make_float4(f * u.x, f * u.y, f * u.z, f * u.w);
            }
            cp_async_wait<0>();
            __syncthreads();                // W is done with; u and the keys are there
            ask_w(c + 1);
            {
                Tile<4> acc;
                acc.clear();
                float* mine = ks + share * SHARE * LDR;
                rows_product<64, 8>(acc, mine + sy * 4, LDR, us + share * SHARE * LDC + x * 4, LDC, SHARE);
                asm volatile("bar.sync %0, 64;" ::"r"(share + 1) : "memory");       // the other warp of the share has read its operand, too
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    *reinterpret_cast<float4*>(mine + at(i / 4 * 64 + sy * 4 + i % 4, x)) = make_float4(acc.at(i, 0), acc.at(i, 1), acc.at(i, 2), acc.at(i, 3));
            }
            __syncthreads();
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int e = (tid >> 2) + i * 64;
                float4 s = *reinterpret_cast<const float4*>(ks + at(e, x));
#pragma unroll
                for (int w = 1; w < CHUNK / SHARE; ++w) {
                    const float4 o = *reinterpret_cast<const float4*>(ks + w * SHARE * LDR + at(e, x));
                    s.x += o.x; s.y += o.y; s.z += o.z; s.w += o.w;
                }
                float4* to = reinterpret_cast<float4*>(st + e * LDC + x * 4);
                const float4 v = *to;
                *to = make_float4(fmaf(whole, v.x, s.x), fmaf(whole, v.y, s.y), fmaf(whole, v.z, s.z), fmaf(whole, v.w, s.w));
            }
            __syncthreads();                // the keys are done with, the state has moved on
            ask_k(c + 1);
        }
        for (int i = tid; i < WC * D / 4; i += WALK_THREADS) {
            const int c = i / (D / 4), e = i % (D / 4) * 4;
            *reinterpret_cast<float4*>(S + c * D + e) = make_float4(st[e * LDC + c], st[(e + 1) * LDC + c], st[(e + 2) * LDC + c], st[(e + 3) * LDC + c]);
        }
        cp_async_wait<0>();
    }
    pdl_trigger();
}

template <int>
__global__ __launch_bounds__(OUTPUT_THREADS, 2) void delta_chunk_outputs(const float* __restrict__ act, float* __restrict__ scratch, float* __restrict__ out, Seqs sq,
                                                                         int n_seqs, Shape z) {
    extern __shared__ __align__(16) float smem[];
    float* qt = smem;                       // [entry][token + 4]
    float* st = qt + D * LDT;               // [entry][column + 4]
    float* pt = st + D * LDT;               // [key][query + 4]
    float* us = pt + CHUNK * LDT;           // [token][column + 4]
    pdl_wait();
    const int2 rows = chunk_rows(sq, n_seqs, blockIdx.x);
    if (rows.y > 0) {
        const int h = blockIdx.y, v0 = blockIdx.z * VT, hq = h / (z.nh / z.n_qk), n = rows.y, dv = z.dv;
        const size_t AW = act_width<HEAD_DECAY>(z);
        const Unit m(scratch, (size_t)blockIdx.x * z.nh + h, dv);
        for (int i = threadIdx.x; i < D * VT / 4; i += OUTPUT_THREADS) cp_async16(st + i / (VT / 4) * LDT + i % (VT / 4) * 4, m.s + (size_t)(i / (VT / 4)) * dv + v0 + i % (VT / 4) * 4, true);
        for (int i = threadIdx.x; i < CHUNK * CHUNK / 4; i += OUTPUT_THREADS) cp_async16(pt + i / (CHUNK / 4) * LDT + i % (CHUNK / 4) * 4, m.p + i * 4, true);
        cp_async_commit();
        // (the weights of later tokens are zeros, and a zero times what is not finite would reach tokens that came before it)
        auto stage_u = [&](bool finite) {
            bool met = false;
            for (int i = threadIdx.x; i < CHUNK * VT / 4; i += OUTPUT_THREADS) {
                const int r = i / (VT / 4), c = i % (VT / 4) * 4;
                float4 v = load_quad(m.u + (size_t)r * dv + v0 + c);
                if (finite) {
                    met |= !(fabsf(v.x) < INFINITY && fabsf(v.y) < INFINITY && fabsf(v.z) < INFINITY && fabsf(v.w) < INFINITY);
                    v.x = fabsf(v.x) < INFINITY ? v.x : 0.f; v.y = fabsf(v.y) < INFINITY ? v.y : 0.f;
                    v.z = fabsf(v.z) < INFINITY ? v.z : 0.f; v.w = fabsf(v.w) < INFINITY ? v.w : 0.f;
                }
                *reinterpret_cast<float4*>(us + r * LDT + c) = v;
            }
            return met;
        };
        const bool met = stage_u(true);
        stage_turned<OUTPUT_THREADS>(qt, act + rows.x * AW + z.q_at + hq * D, AW, n);
        cp_async_wait<0>();
        const bool spoilt = __syncthreads_or(met);
        const int ty = thread_row(threadIdx.x), tx = thread_col(threadIdx.x);
        Tile<4> acc;
        acc.clear();
        product<4, 8>(acc, qt, LDT, st, LDT, D, ty, tx);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 f = *reinterpret_cast<const float2*>(m.grow + i / 2 * 32 + ty * 4 + i % 2 * 2);
            acc.scale(i, f.x, f.y);
        }
        product<4, 8>(acc, pt, LDT, us, LDT, (n + 7) & ~7, ty, tx);
        float* dst = out + (size_t)rows.x * z.nh * dv + h * dv + v0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int q = i / 4 * 32 + ty * 4 + i % 4;
            if (q < n) *reinterpret_cast<float4*>(dst + (size_t)q * z.nh * dv + tx * 4) = make_float4(acc.at(i, 0), acc.at(i, 1), acc.at(i, 2), acc.at(i, 3));
        }
        if (spoilt) {           // values that are not finite, for the tokens from theirs on
            __syncthreads();
            stage_u(false);
            __syncthreads();
#pragma unroll 1
            for (int i = threadIdx.x; i < n * VT; i += OUTPUT_THREADS) {
                const int q = i / VT, c = i % VT;
                float more = 0.f;
#pragma unroll 1
                for (int k = 0; k <= q; ++k) {
                    const float v = us[k * LDT + c];
                    if (!(fabsf(v) < INFINITY)) more = fmaf(pt[k * LDT + q], v, more);
                }
                if (more != 0.f) dst[(size_t)q * z.nh * dv + c] += more;      // (after the block's barriers)
            }
        }
    }
    pdl_trigger();
}
}  // namespace wide
}  // namespace convrec
