// The decayed linear recurrence of lightning_attention.cu over prompts, 64 tokens at a time:
//
//   S_t = g S_(t-1) + k_t v_t^T ;  o_t = S_t^T q_t          (g a constant a head, S [d, dv] per request and head)
//
// With S before a chunk of n tokens and i, j counted inside it,
//
//   o_i = g^(i+1) S^T q_i + sum_{j <= i} g^(i-j) (q_i . k_j) v_j ;   S <- g^n S + sum_j g^(n-1-j) k_j v_j^T
//
// which is the recurrence written out.  The walk token by token offers one request 1,024 warps, each bound by its own
// chain of tokens (2,048 tokens, 16 heads of 128 x 128: 283 us after a pass of 26 for silu); here all chunks are worked on at once, as small
// products of 64 rows, and only an elementwise pass goes from chunk to chunk:
//
//   chunk_update:  (chunk, head, 64 columns of v)  U = sum_j g^(n-1-j) v_j k_j^T
//   chunk_states:  (request, head, 4 entries a thread)  walks the request's chunks: U is replaced by the state before the
//                  chunk, the slot's state by the one after the last
//   chunk_outputs: (chunk, head, 64 columns of v)  the scores of the chunk's tokens against each other, decayed, times v,
//                  and the read-out of the state before the chunk
//
// Everything is float32 (FFMA, two at a time), as in the walk; powers of g are made in float64 and rounded once, where the walk
// rounds at every token.  Bound by the FMA pipes and by reads of shared memory: a thread has 8 x 4 or 8 x 8 outputs, so
// three or four 16-byte reads feed 32 or 64 FMAs.  200 us (43, 25 and 132; 47, 25 and 151 with pairs of columns in the FMAs) at the sizes above, silu
// included (inputs are activated on their way into shared memory).
#include "chunk_products.cuh"

namespace {
using namespace chunkprod;
constexpr int VT = 64, THREADS = 128;

__device__ __forceinline__ float silu_f(float z) { return z / (1.0f + expf(-z)); }

struct Rows {
    const void* x;              // rows of q | k | v, `stride` elements apart
    long long stride;
    int q_off, k_off, v_off;
};
struct Seqs {
    const int* cu_seqlens;
    const int* ctx_lens;
    const int* state_slots;
    int n_seqs;
};
// Chunk c of the step: its first token's row and its tokens (none: there is no such chunk).
__device__ __forceinline__ int2 chunk_rows(const Seqs& s, int c) {
    for (int b = 0; b < s.n_seqs; ++b) {
        const int row = s.cu_seqlens[b], n = s.cu_seqlens[b + 1] - row, chunks = (n + CHUNK - 1) / CHUNK;
        if (c < chunks) return make_int2(row + c * CHUNK, min(CHUNK, n - c * CHUNK));
        c -= chunks;
    }
    return make_int2(0, 0);
}
// g^n, rounded once.
__device__ __forceinline__ float power(float g, int n) {
    double r = 1.0, b = g;
    for (; n > 0; n >>= 1, b *= b)
        if (n & 1) r *= b;
    return (float)r;
}

// Eight (bf16) or four (float) entries of a row, activated.
template <typename T, bool SILU> __device__ __forceinline__ void load_piece(const T* p, bool valid, float (&v)[16 / sizeof(T)]) {
    constexpr int N = 16 / sizeof(T);
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = 0.f;
    if (valid) {
        load16<T>(p, v);
        if (SILU) {
#pragma unroll
            for (int i = 0; i < N; ++i) v[i] = silu_f(v[i]);
        }
    }
}

// rows x cols of x into shared memory as they lie, [row][cols + 4]; rows from n on become zeros; `scale` a row.  FINITE: what is
// not finite becomes 0 there; whether this thread met some.
template <typename T, bool SILU, int COLS, bool FINITE = false, typename Scale>
__device__ __forceinline__ bool stage(float* dst, const T* x, long long stride, int n, Scale scale) {
    constexpr int N = 16 / sizeof(T), P = COLS / N;
    bool spoilt = false;
#pragma unroll 4
    for (int i = threadIdx.x; i < CHUNK * P; i += THREADS) {
        const int r = i / P, c = i % P * N;
        float v[N];
        load_piece<T, SILU>(x + (size_t)r * stride + c, r < n, v);
        if (FINITE) {
#pragma unroll
            for (int u = 0; u < N; ++u) {
                const bool finite = fabsf(v[u]) < INFINITY;
                spoilt |= !finite;
                v[u] = finite ? v[u] : 0.f;
            }
        }
        const float f = scale(r);
#pragma unroll
        for (int u = 0; u < N; u += 4)
            *reinterpret_cast<float4*>(dst + r * (COLS + 4) + c + u) = make_float4(v[u] * f, v[u + 1] * f, v[u + 2] * f, v[u + 3] * f);
    }
    return spoilt;
}
// The same turned: [col][64 rows + 4].  A warp takes 16 rows x 2 pieces (bf16) or 8 x 4 (float): whole sectors of memory, and
// no more than two of its writes in a bank.
template <typename T, bool SILU, int COLS>
__device__ __forceinline__ void stage_turned(float* dst, const T* x, long long stride, int n) {
    constexpr int N = 16 / sizeof(T), P = COLS / N, RW = sizeof(T) == 2 ? 16 : 8, PW = 32 / RW;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll 4
    for (int i = warp; i < CHUNK / RW * (P / PW); i += THREADS / 32) {
        const int r = i % (CHUNK / RW) * RW + lane % RW, c = (i / (CHUNK / RW) * PW + lane / RW) * N;
        float v[N];
        load_piece<T, SILU>(x + (size_t)r * stride + c, r < n, v);
#pragma unroll
        for (int u = 0; u < N; ++u) dst[(c + u) * LDT + r] = v[u];
    }
}

template <typename T, bool SILU, int D>
__global__ __launch_bounds__(THREADS) void chunk_update_kernel(const Rows in, float* __restrict__ states, const float* __restrict__ decay,
                                                               const Seqs seqs, int nh, int dv) {
    extern __shared__ __align__(16) float smem[];
    pdl_wait();
    const int2 rows = chunk_rows(seqs, blockIdx.x);
    if (rows.y > 0) {
        const int h = blockIdx.y, v0 = blockIdx.z * VT, n = rows.y;
        float* vs = smem;                                  // [token][VT + 4]
        float* ks = vs + CHUNK * (VT + 4);                 // [token][D + 4], decayed to the chunk's end
        const T* x = reinterpret_cast<const T*>(in.x) + (size_t)rows.x * in.stride;
        const float g = decay[h];
        __shared__ float pw[CHUNK];
        if (threadIdx.x < CHUNK) pw[threadIdx.x] = power(g, max(0, n - 1 - (int)threadIdx.x));
        __syncthreads();
        stage<T, SILU, VT>(vs, x + in.v_off + h * dv + v0, in.stride, n, [](int) { return 1.0f; });
        stage<T, SILU, D>(ks, x + in.k_off + h * D, in.stride, n, [&](int r) { return pw[r]; });
        __syncthreads();
        const int ty = thread_row(threadIdx.x), tx = thread_col(threadIdx.x);
        Tile<D / 16> acc;
        acc.clear();
        product<D / 16, 0>(acc, vs, VT + 4, ks, D + 4, n, ty, tx);
        float* out = states + (((size_t)blockIdx.x * nh + h) * dv + v0) * D;
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < D / 16; j += 4)
                *reinterpret_cast<float4*>(out + (size_t)(i / 4 * 32 + ty * 4 + i % 4) * D + j * 16 + tx * 4) =
                    make_float4(acc.at(i, j), acc.at(i, j + 1), acc.at(i, j + 2), acc.at(i, j + 3));
    }
    pdl_trigger();
}

__global__ __launch_bounds__(256) void chunk_states_kernel(float4* __restrict__ states, float4* __restrict__ state, const float* __restrict__ decay,
                                                           const Seqs seqs, int nh, int quads) {
    pdl_wait();
    const int b = blockIdx.x, h = blockIdx.y, at = blockIdx.z * 256 + threadIdx.x;
    int before = 0;
    for (int o = 0; o < b; ++o) before += (seqs.cu_seqlens[o + 1] - seqs.cu_seqlens[o] + CHUNK - 1) / CHUNK;
    const int n = seqs.cu_seqlens[b + 1] - seqs.cu_seqlens[b], chunks = (n + CHUNK - 1) / CHUNK;
    if (at < quads && n > 0) {
        const float g = decay[h], whole = power(g, CHUNK), last = power(g, n - (chunks - 1) * CHUNK);
        float4* slot = state + ((size_t)seqs.state_slots[b] * nh + h) * quads + at;
        float4 s = seqs.ctx_lens[b] - n == 0 ? make_float4(0.f, 0.f, 0.f, 0.f) : *slot;        // (a request that starts here starts from zero)
        float4* u = states + ((size_t)before * nh + h) * quads + at;
        const size_t step = (size_t)nh * quads;
#pragma unroll 8
        for (int c = 0; c < chunks; ++c, u += step) {
            const float4 x = *u;
            *u = s;
            const float f = c == chunks - 1 ? last : whole;
            s = make_float4(fmaf(f, s.x, x.x), fmaf(f, s.y, x.y), fmaf(f, s.z, x.z), fmaf(f, s.w, x.w));
        }
        *slot = s;
    }
    pdl_trigger();
}

template <typename T, bool SILU, int D>
__global__ __launch_bounds__(THREADS) void chunk_outputs_kernel(const Rows in, const float* __restrict__ states, float* __restrict__ out,
                                                                const float* __restrict__ decay, const Seqs seqs, int nh, int dv) {
    extern __shared__ __align__(16) float smem[];
    pdl_wait();
    const int2 rows = chunk_rows(seqs, blockIdx.x);
    if (rows.y > 0) {
        const int h = blockIdx.y, v0 = blockIdx.z * VT, n = rows.y;
        float* qt = smem;                        // [entry][token + 4]
        float* xt = qt + D * LDT;                // keys, then the state before the chunk, [entry][token or column + 4]
        float* vs = xt + D * LDT;                // [token][VT + 4]
        float* pt = vs + CHUNK * (VT + 4);       // decayed scores, [key token][query token + 4]
        const T* x = reinterpret_cast<const T*>(in.x) + (size_t)rows.x * in.stride;
        const float g = decay[h];
        __shared__ float pw[CHUNK + 1];
        if (threadIdx.x <= CHUNK) pw[threadIdx.x] = power(g, threadIdx.x);
        stage_turned<T, SILU, D>(qt, x + in.q_off + h * D, in.stride, n);
        stage_turned<T, SILU, D>(xt, x + in.k_off + h * D, in.stride, n);
        // (the weights of later keys are zeros, and a zero times what is not finite would reach tokens that came before it)
        const bool met = stage<T, SILU, VT, true>(vs, x + in.v_off + h * dv + v0, in.stride, n, [](int) { return 1.0f; });
        const bool spoilt = __syncthreads_or(met);
        const int ty = thread_row(threadIdx.x), tx = thread_col(threadIdx.x);
        Tile<4> acc;
        acc.clear();
        product<4, 8>(acc, qt, LDT, xt, LDT, D, ty, tx);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int q = i / 4 * 32 + ty * 4 + i % 4;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int k = tx * 4 + j;
                pt[k * LDT + q] = q >= k ? acc.at(i, j) * pw[q - k] : 0.f;
            }
        }
        __syncthreads();
        stage_turned<float, false, D>(xt, states + (((size_t)blockIdx.x * nh + h) * dv + v0) * D, D, VT);
        __syncthreads();
        acc.clear();
        product<4, 8>(acc, qt, LDT, xt, LDT, D, ty, tx);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int q = i / 2 * 32 + ty * 4 + i % 2 * 2;
            acc.scale(i, pw[q + 1], pw[q + 2]);
        }
        product<4, 8>(acc, pt, LDT, vs, VT + 4, (n + 7) & ~7, ty, tx);     // (rows of zeros beyond n)
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int q = i / 4 * 32 + ty * 4 + i % 4;
            if (q < n)
                *reinterpret_cast<float4*>(out + (size_t)(rows.x + q) * nh * dv + h * dv + v0 + tx * 4) = make_float4(acc.at(i, 0), acc.at(i, 1), acc.at(i, 2), acc.at(i, 3));
        }
        if (spoilt) {           // values that are not finite, for the tokens from theirs on
            __syncthreads();
            stage<T, SILU, VT>(vs, x + in.v_off + h * dv + v0, in.stride, n, [](int) { return 1.0f; });
            __syncthreads();
#pragma unroll 1
            for (int i = threadIdx.x; i < n * VT; i += THREADS) {
                const int q = i / VT, c = i % VT;
                float more = 0.f;
#pragma unroll 1
                for (int k = 0; k <= q; ++k) {
                    const float v = vs[k * (VT + 4) + c];
                    if (!(fabsf(v) < INFINITY)) more = fmaf(pt[k * LDT + q], v, more);
                }
                if (more != 0.f) out[(size_t)(rows.x + q) * nh * dv + h * dv + v0 + c] += more;      // (after the block's barriers)
            }
        }
    }
    pdl_trigger();   // the next kernel of the stream may start its launch
}

template <typename T, bool SILU, int D>
int run(const Rows& in, float* out, float* states, float* state, const float* decay, const Seqs& seqs, int chunks, int nh, int dv, cudaStream_t stream) {
    constexpr int update_smem = CHUNK * (VT + 4 + D + 4) * 4, output_smem = (2 * D * LDT + CHUNK * (VT + 4) + CHUNK * LDT) * 4;
    cudaError_t e = cudaFuncSetAttribute(chunk_update_kernel<T, SILU, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, update_smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(chunk_outputs_kernel<T, SILU, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, output_smem);
    if (e != cudaSuccess) return (int)e;
    const dim3 grid(chunks, nh, dv / VT);
    rlis_launch(chunk_update_kernel<T, SILU, D>, grid, THREADS, update_smem, stream, in, states, decay, seqs, nh, dv);
    const int quads = dv * D / 4;
    rlis_launch(chunk_states_kernel, dim3(seqs.n_seqs, nh, (quads + 255) / 256), 256, 0, stream, reinterpret_cast<float4*>(states),
                reinterpret_cast<float4*>(state), decay, seqs, nh, quads);
    rlis_launch(chunk_outputs_kernel<T, SILU, D>, grid, THREADS, output_smem, stream, in, states, out, decay, seqs, nh, dv);
    return RLIS_LAUNCH_CHECK();
}
}  // namespace

extern "C" int rlis_lightning_chunk_tokens(void) { return CHUNK; }
extern "C" int rlis_lightning_chunks_takes(int d, int dv) { return (d == 64 || d == 128) && dv > 0 && dv % VT == 0; }

// The contract of rlis_lightning_scan (silu) and, without `silu`, of rlis_recurrence_scan with a decay a head.  `states`: float32
// [chunks, nh, dv, d], chunks at least the sum over the requests of their tokens / 64, rounded up.
extern "C" int rlis_lightning_chunks(const void* rows, long long stride, int q_off, int k_off, int v_off, float* out, float* states, float* state,
                                     const float* decay, const int* cu_seqlens, const int* ctx_lens, const int* state_slots, int n_seqs, int chunks,
                                     int nh, int d, int dv, int silu, int dtype, cudaStream_t stream) {
    if (n_seqs <= 0 || chunks <= 0) return 0;
    if (!rlis_lightning_chunks_takes(d, dv) || nh <= 0 || nh > 65535 || dv / VT > 65535) return RLIS_ERR_UNSUPPORTED;
    const int vec = dtype == RLIS_BF16 ? 8 : 4;
    if (stride % vec || q_off % vec || k_off % vec || v_off % vec ||
        ((reinterpret_cast<uintptr_t>(rows) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(states) | reinterpret_cast<uintptr_t>(state)) & 15))
        return RLIS_ERR_UNSUPPORTED;
    const Rows in = {rows, stride, q_off, k_off, v_off};
    const Seqs seqs = {cu_seqlens, ctx_lens, state_slots, n_seqs};
#define RLIS_CHUNKS(T, S) (d == 64 ? run<T, S, 64>(in, out, states, state, decay, seqs, chunks, nh, dv, stream) \
                                   : run<T, S, 128>(in, out, states, state, decay, seqs, chunks, nh, dv, stream))
    if (dtype == RLIS_BF16) return silu ? RLIS_CHUNKS(bf16, true) : RLIS_ERR_UNSUPPORTED;
    if (dtype == RLIS_F32) return silu ? RLIS_CHUNKS(float, true) : RLIS_CHUNKS(float, false);
#undef RLIS_CHUNKS
    return RLIS_ERR_UNSUPPORTED;
}
