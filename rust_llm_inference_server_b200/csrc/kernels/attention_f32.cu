// Causal grouped-query attention of the float32 path over the paged cache, for head sizes that are multiples of 16 up to
// 128 and groups of up to 8 query heads (attention_generic.cu takes the others).  Scores, softmax and the value sum
// are float32, as there.
//
// The keys of a request are cut at multiples of PIECE = 256, whatever the step: inside a piece a query walks blocks of
// 32 keys that start at multiples of 32 with a running maximum, and the pieces are then folded together in their
// order.  So a token's sums are taken in an order that depends on its position alone, and the same token gives
// the same bits as a single token, whose pieces are taken by different CTAs, and inside a prompt, where
// a CTA takes all of them.
//
// A CTA takes one key/value head and the query heads of its group; blocks of keys and values come into shared memory by
// 16-byte asynchronous copies, once for all of them.
//   single tokens (SPLIT): a CTA a (request, kv head, piece), a warp a query head; a second kernel folds the pieces.  Bound
//     by the cache's bytes: a group of four heads reads them once where the kernel with a warp a head read them four
//     times, and a context of 2,048 offers eight times as many CTAs.  The pieces that exist stand one after the other, request by
//     request, and a CTA looks its own up from the positions, so that neither launch nor scratch memory is sized by the longest context
//     times the requests (64 requests of 200 keys beside one of 131,072, 32 heads of 128: 545 MB by the longest, 17 by the pieces).  Beyond
//     SPLIT_ROWS requests, which are many waves of CTAs by themselves, a CTA takes a whole context.
//   prompts: 8 warps of R = 4 rows, a row a (token, query head); lanes are keys for the scores and dimensions for
//     the value sum, so a key's 16 bytes in shared memory serve four rows.  The weights of a block go through shared memory, four rows' in a
//     read: 700 tokens, 32 heads of 64 157 us, with a shuffle a key and row 175 (eight rows a warp 225: half as many CTAs, whose longest rows are
//     the kernel's end).
#include "common.cuh"
#include "mma_utils.cuh"
#include <math.h>

namespace {
constexpr int PIECE = 256, BLOCK = 32, PROMPT_WARPS = 8, PROMPT_ROWS = 4, MAX_GROUP = 8, STAGES = 3, SPLIT_ROWS = 1024;

struct Args {
    const float* q;
    const float* k_cache;
    const float* v_cache;
    float* out;
    float* partial;               // [pieces of all rows, nh, d + 2]: value sum, maximum, denominator of a piece
    const int* seq_of_token;
    const int* positions;
    const int* block_tables;
    const int* token_rows;        // the step's tokens this launch computes, or null for all
    int max_blocks, n_rows, tokens_per_cta, slots, nh, nkv, d, page_size;
    float scale;
    int window;
};

__device__ __forceinline__ int first_key(int pos, int window) { return window > 0 ? max(0, pos - window + 1) : 0; }
__device__ __forceinline__ int row_token_of(const Args& p, int row) { return p.token_rows != nullptr ? p.token_rows[row] : row; }
__device__ __forceinline__ int row_pieces(const Args& p, int row) {
    const int pos = p.positions[row_token_of(p, row)];
    return pos / PIECE - first_key(pos, p.window) / PIECE + 1;
}

// Whose piece number `slot` is, and which of that row's it is: all threads of the block; row -1 beyond the last.
__device__ __forceinline__ int2 piece_at(const Args& p, int slot) {
    __shared__ int totals[MAX_GROUP];
    __shared__ int2 found;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, per = (p.n_rows + blockDim.x - 1) / blockDim.x;
    const int row0 = tid * per, row1 = min(row0 + per, p.n_rows);
    int own = 0;
#pragma unroll 4
    for (int row = row0; row < row1; ++row) own += row_pieces(p, row);
    int incl = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int n = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += n;
    }
    if (lane == 31) totals[warp] = incl;
    if (tid == 0) found = make_int2(-1, 0);
    __syncthreads();
    int before = incl - own;
    for (int w = 0; w < warp; ++w) before += totals[w];
    if (slot >= before && slot < before + own) {
        int row = row0, at = slot - before;
        for (int n; at >= (n = row_pieces(p, row)); ++row) at -= n;
        found = make_int2(row, at);
    }
    __syncthreads();
    return found;
}

// What scores are taken from before expf: their running maximum, or 0 while all of them are -inf (whose weights are 0 then, not the NaN
// of -inf - -inf).
__device__ __forceinline__ float reference_score(float top) { return top == -INFINITY ? 0.f : top; }

// Folds the piece (m, l, a) into the ones before it (M, L, A).
template <int DL> __device__ __forceinline__ void fold(float& M, float& L, float (&A)[DL], float m, float l, const float (&a)[DL]) {
    const float top = fmaxf(M, m), from = reference_score(top), c0 = expf(M - from), c1 = expf(m - from);
    L = __fmaf_rn(L, c0, __fmul_rn(l, c1));
#pragma unroll
    for (int i = 0; i < DL; ++i) A[i] = __fmaf_rn(A[i], c0, __fmul_rn(a[i], c1));
    M = top;
}

template <int DL, int R, bool SPLIT>
__global__ __launch_bounds__((SPLIT ? MAX_GROUP : PROMPT_WARPS) * 32) void attn_f32_kernel(const Args p) {
    static_assert(R == 1 || R % 4 == 0, "weights go by fours");
    extern __shared__ __align__(16) float smem[];
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const int group = p.nh / p.nkv, kvh = SPLIT ? blockIdx.y : blockIdx.x, d = p.d, ld = d + 4;
    float* qs = smem + warp * R * d;                                        // this warp's rows of q
    float* ring = smem + warps * R * d;
    const int stage_floats = 2 * BLOCK * ld;
    int* mapped = reinterpret_cast<int*>(ring + STAGES * stage_floats);     // [stage][key]: whether its page is there
    float* ws = reinterpret_cast<float*>(mapped + STAGES * BLOCK) + warp * BLOCK * R;       // [key][row] weights of a block (R > 1)
    const int2 piece = SPLIT ? piece_at(p, blockIdx.x) : make_int2(0, 0);
    if (SPLIT && piece.x < 0) return;
    // long tiles first: the last tokens of a prompt see the most keys
    const int t0 = SPLIT ? piece.x : (gridDim.y - 1 - blockIdx.y) * p.tokens_per_cta;
    const int nt = SPLIT ? 1 : min(p.tokens_per_cta, p.n_rows - t0);
    auto token = [&](int i) { return row_token_of(p, t0 + i); };

    // this warp's rows: token of the tile and query head
    int row_token[R], row_head[R], row_pos[R], row_lo[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int row = warp * R + r, ti = row / group;
        const bool there = ti < nt;
        row_token[r] = there ? ti : -1;
        row_head[r] = kvh * group + row % group;
        const int t = token(there ? ti : 0);
        row_pos[r] = p.positions[t];
        row_lo[r] = first_key(row_pos[r], p.window);
        const float* src = p.q + ((size_t)t * p.nh + row_head[r]) * d;
        for (int j = lane; j < d; j += 32) qs[r * d + j] = src[j];
    }
    __syncwarp();

    // tokens of one request at a time (a tile of a mixed step may hold the end of one portion and the start of the next)
    for (int s0 = 0; s0 < nt;) {
        const int seq = p.seq_of_token[token(s0)];
        int s1 = s0, last = 0, lo = 0x7fffffff;
        for (; s1 < nt && p.seq_of_token[token(s1)] == seq; ++s1) {
            const int pos = p.positions[token(s1)];
            last = max(last, pos);
            lo = min(lo, first_key(pos, p.window));
        }
        const int* table = p.block_tables + (size_t)seq * p.max_blocks;
        int kb0 = lo & ~(BLOCK - 1), end = last + 1;            // keys kb0 .. end - 1, block by block
        const int piece0 = lo / PIECE, pieces = last / PIECE - piece0 + 1;
        if (SPLIT) {
            kb0 = max(kb0, (piece0 + piece.y) * PIECE);
            end = min(end, (piece0 + piece.y + 1) * PIECE);
        }
        const int blocks = (end - kb0 + BLOCK - 1) / BLOCK;

        // a key's row of keys and of values is copied by `warps` neighbouring threads; its page is looked up a block ahead
        const int key_row = threadIdx.x / warps, part = threadIdx.x % warps;
        auto page_of = [&](int b) {
            const int key = kb0 + b * BLOCK + key_row;
            return b < blocks && key < end ? table[key / p.page_size] : -1;
        };
        int next_page = page_of(0);
        auto request = [&](int b) {
            if (b < blocks) {
                const int key = kb0 + b * BLOCK + key_row, page = next_page;
                next_page = page_of(b + 1);
                float* kd = ring + (b % STAGES) * stage_floats + key_row * ld;
                float* vd = kd + BLOCK * ld;
                const size_t off = page >= 0 ? (((size_t)page * p.nkv + kvh) * p.page_size + key % p.page_size) * d : 0;
                for (int c = part * 4; c < d; c += warps * 4) {
                    cp_async16(kd + c, p.k_cache + off + c, page >= 0);
                    cp_async16(vd + c, p.v_cache + off + c, page >= 0);
                }
                if (part == 0) mapped[(b % STAGES) * BLOCK + key_row] = page >= 0;
            }
            cp_async_commit();
        };
        __syncthreads();                // (the ring of the request before this one is free)
#pragma unroll
        for (int b = 0; b < STAGES - 1; ++b) request(b);

        float m[R], l[R], acc[R][DL], M[R], L[R], A[R][DL];
        bool begun[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            m[r] = -INFINITY;
            l[r] = 0.f;
            M[r] = L[r] = 0.f;
            begun[r] = false;
#pragma unroll
            for (int i = 0; i < DL; ++i) acc[r][i] = A[r][i] = 0.f;
        }
        for (int b = 0; b < blocks; ++b) {
            cp_async_wait<STAGES - 2>();
            __syncthreads();
            request(b + STAGES - 1);
            const float* ks = ring + (b % STAGES) * stage_floats;
            const float* vs = ks + BLOCK * ld;
            const int kb = kb0 + b * BLOCK, key = kb + lane;
            bool live[R], any = false;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                live[r] = row_token[r] >= s0 && row_token[r] < s1 && kb <= row_pos[r] && kb + BLOCK > row_lo[r];     // uniform over the warp
                any |= live[r];
            }
            if (any) {
                float s[R];
#pragma unroll
                for (int r = 0; r < R; ++r) s[r] = 0.f;
                for (int j = 0; j < d; j += 4) {
                    const float4 kv = *reinterpret_cast<const float4*>(ks + lane * ld + j);
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const float4 qv = *reinterpret_cast<const float4*>(qs + r * d + j);
                        s[r] = fmaf(qv.x, kv.x, s[r]);
                        s[r] = fmaf(qv.y, kv.y, s[r]);
                        s[r] = fmaf(qv.z, kv.z, s[r]);
                        s[r] = fmaf(qv.w, kv.w, s[r]);
                    }
                }
                const bool there = mapped[(b % STAGES) * BLOCK + lane] != 0;
                float w[R];
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    w[r] = 0.f;
                    if (!live[r]) continue;
                    const bool valid = key >= row_lo[r] && key <= row_pos[r];
                    // a page the host did not map: make it visible
                    const float sc = !valid ? -INFINITY : there ? __fmul_rn(s[r], p.scale) : NAN;
                    const float m_new = fmaxf(m[r], warp_max(sc)), from = reference_score(m_new);
                    w[r] = valid ? expf(sc - from) : 0.f;
                    const float corr = expf(m[r] - from);
                    l[r] = __fmaf_rn(l[r], corr, warp_sum(w[r]));
#pragma unroll
                    for (int i = 0; i < DL; ++i) acc[r][i] *= corr;
                    m[r] = m_new;
                }
                // p . v in the order of the keys; a key without weight takes part with nothing, whatever its row holds
                if (R > 1) {
#pragma unroll
                    for (int r = 0; r < R; r += 4) *reinterpret_cast<float4*>(ws + lane * R + r) = make_float4(w[r], w[(r + 1) % R], w[(r + 2) % R], w[(r + 3) % R]);
                    __syncwarp();
                }
#pragma unroll 8
                for (int kk = 0; kk < BLOCK; ++kk) {
                    float v[DL], pk[R];
#pragma unroll
                    for (int i = 0; i < DL; ++i) v[i] = lane + 32 * i < d ? vs[kk * ld + lane + 32 * i] : 0.f;
                    if (R > 1) {
#pragma unroll
                        for (int r = 0; r < R; r += 4) *reinterpret_cast<float4*>(pk + r) = *reinterpret_cast<const float4*>(ws + kk * R + r);
                    } else {
                        pk[0] = __shfl_sync(0xffffffffu, w[0], kk);
                    }
#pragma unroll
                    for (int r = 0; r < R; ++r) {
#pragma unroll
                        for (int i = 0; i < DL; ++i) acc[r][i] = pk[r] != 0.f ? fmaf(pk[r], v[i], acc[r][i]) : acc[r][i];
                    }
                }
                if (R > 1) __syncwarp();            // (the weights have been read before the next block's)
            }
            if (!SPLIT && ((kb + BLOCK) % PIECE == 0 || b == blocks - 1)) {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    if (m[r] == -INFINITY && l[r] == 0.f) continue;             // the row sees nothing of this piece, or only scores of -inf
                    if (begun[r]) {
                        fold<DL>(M[r], L[r], A[r], m[r], l[r], acc[r]);
                    } else {
                        begun[r] = true;
                        M[r] = m[r];
                        L[r] = l[r];
#pragma unroll
                        for (int i = 0; i < DL; ++i) A[r][i] = acc[r][i];
                    }
                    m[r] = -INFINITY;
                    l[r] = 0.f;
#pragma unroll
                    for (int i = 0; i < DL; ++i) acc[r][i] = 0.f;
                }
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (row_token[r] < s0 || row_token[r] >= s1) continue;
            if (SPLIT && pieces > 1 && p.partial != nullptr) {
                float* dst = p.partial + ((size_t)blockIdx.x * p.nh + row_head[r]) * (d + 2);
#pragma unroll
                for (int i = 0; i < DL; ++i)
                    if (lane + 32 * i < d) dst[lane + 32 * i] = acc[r][i];
                if (lane == 0) { dst[d] = m[r]; dst[d + 1] = l[r]; }
                continue;
            }
            float* orow = p.out + ((size_t)token(row_token[r]) * p.nh + row_head[r]) * d;
            const float inv = 1.0f / (SPLIT ? l[r] : L[r]);
#pragma unroll
            for (int i = 0; i < DL; ++i)
                if (lane + 32 * i < d) orow[lane + 32 * i] = (SPLIT ? acc[r][i] : A[r][i]) * inv;
        }
        s0 = s1;
    }
    pdl_trigger();   // the next kernel of the stream may start its launch
}

// One warp a (token, query head): its pieces in their order.
template <int DL> __global__ __launch_bounds__(128) void attn_f32_fold_kernel(const Args p) {
    pdl_wait();
    const int lane = threadIdx.x & 31, row = blockIdx.x * 4 + (threadIdx.x >> 5), d = p.d;
    if (row < p.n_rows * p.nh) {
        const int i = row / p.nh, t = row_token_of(p, i), pieces = row_pieces(p, i);
        if (pieces > 1) {
            int slot = 0;                   // of its first piece
            for (int o = lane; o < i; o += 32) slot += row_pieces(p, o);
            slot = __reduce_add_sync(0xffffffffu, slot);
            if (slot + pieces > p.slots) return;            // (the host counts them; never read beyond what it made room for)
            const size_t step = (size_t)p.nh * (d + 2);
            const float* src = p.partial + slot * step + (size_t)(row % p.nh) * (d + 2);
            float M = 0.f, L = 0.f, A[DL];
            for (int z = 0; z < pieces; ++z, src += step) {
                float a[DL];
#pragma unroll
                for (int u = 0; u < DL; ++u) a[u] = lane + 32 * u < d ? src[lane + 32 * u] : 0.f;
                const float m = src[d], l = src[d + 1];
                if (z == 0) {
                    M = m;
                    L = l;
#pragma unroll
                    for (int u = 0; u < DL; ++u) A[u] = a[u];
                } else {
                    fold<DL>(M, L, A, m, l, a);
                }
            }
            float* orow = p.out + ((size_t)t * p.nh + row % p.nh) * d;
            const float inv = 1.0f / L;
#pragma unroll
            for (int u = 0; u < DL; ++u)
                if (lane + 32 * u < d) orow[lane + 32 * u] = A[u] * inv;
        }
    }
    pdl_trigger();
}

template <int DL> int run(Args p, bool folds, bool single, cudaStream_t stream) {
    const int group = p.nh / p.nkv;
    auto smem = [&](int rows) { return (rows * p.d + STAGES * 2 * BLOCK * (p.d + 4) + rows * BLOCK) * (int)sizeof(float) + STAGES * BLOCK * (int)sizeof(int); };
    if (p.slots > 0) {
        auto kernel = attn_f32_kernel<DL, 1, true>;
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem(MAX_GROUP));
        if (e != cudaSuccess) return (int)e;
        if (p.nkv > 65535) return RLIS_ERR_UNSUPPORTED;
        rlis_launch(kernel, dim3(p.slots, p.nkv), group * 32, smem(group), stream, p);
        if (folds) rlis_launch(attn_f32_fold_kernel<DL>, (p.n_rows * p.nh + 3) / 4, 128, 0, stream, p);
        return RLIS_LAUNCH_CHECK();
    }
    if (single) {
        auto kernel = attn_f32_kernel<DL, 1, false>;
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem(MAX_GROUP));
        if (e != cudaSuccess) return (int)e;
        if (p.n_rows > 65535) return RLIS_ERR_UNSUPPORTED;
        p.tokens_per_cta = 1;
        rlis_launch(kernel, dim3(p.nkv, p.n_rows), group * 32, smem(group), stream, p);
        return RLIS_LAUNCH_CHECK();
    }
    auto kernel = attn_f32_kernel<DL, PROMPT_ROWS, false>;
    constexpr int ROWS = PROMPT_WARPS * PROMPT_ROWS;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem(ROWS));
    if (e != cudaSuccess) return (int)e;
    p.tokens_per_cta = ROWS / group;
    const int tiles = (p.n_rows + p.tokens_per_cta - 1) / p.tokens_per_cta;
    if (tiles > 65535) return RLIS_ERR_UNSUPPORTED;
    rlis_launch(kernel, dim3(p.nkv, tiles), PROMPT_WARPS * 32, smem(ROWS), stream, p);
    return RLIS_LAUNCH_CHECK();
}
}  // namespace

// Keys of a piece, and up to how many single tokens' contexts are cut into them: what the host sizes `partial` by.
extern "C" int rlis_attention_f32_piece(void) { return PIECE; }
extern "C" int rlis_attention_f32_split_rows(void) { return SPLIT_ROWS; }
extern "C" int rlis_attention_f32_takes(int nh, int nkv, int d) {
    return d > 0 && d % 16 == 0 && d <= 128 && nkv > 0 && nh % nkv == 0 && nh / nkv <= MAX_GROUP;
}

// `single` 0: any query lengths, a CTA a tile of tokens.  Otherwise every row is a token on its own: with `slots` their contexts are cut into
// pieces, of which there are at most that many (further CTAs find nothing to do), and `partial` is float32 [slots, nh, d + 2] if some context has
// more than one (`folds`); with 0 slots a CTA takes a whole context.
extern "C" int rlis_attention_f32(const float* q, const float* k_cache, const float* v_cache, float* out, float* partial,
                                  const int* seq_of_token, const int* positions, const int* block_tables, const int* token_rows,
                                  int max_blocks, int n_rows, int single, int slots, int folds, int nh, int nkv, int d, int page_size, float scale,
                                  int window, cudaStream_t stream) {
    if (n_rows <= 0) return 0;
    if (!rlis_attention_f32_takes(nh, nkv, d) || page_size <= 0 || slots < 0 || (slots > 0 && (!single || n_rows > SPLIT_ROWS)) ||
        (folds && (slots == 0 || partial == nullptr)))
        return RLIS_ERR_UNSUPPORTED;
    const Args p = {q, k_cache, v_cache, out, partial, seq_of_token, positions, block_tables, token_rows, max_blocks, n_rows, 1,
                    slots, nh, nkv, d, page_size, scale, window};
    return d <= 32 ? run<1>(p, folds != 0, single != 0, stream) : d <= 64 ? run<2>(p, folds != 0, single != 0, stream) : run<4>(p, folds != 0, single != 0, stream);
}
