// Attention over latents for long portions of prompts, with every head's keys and values formed (bfloat16).
//
// attention_latent_mma.cu scores against the cached rows themselves, [c | k_rot], with the key map folded into the query: 576 +
// 512 multiply-adds a (token, key, head) at a latent of 512 and 64 rotated entries, and nothing to prepare.  Here the context's
// latents go through the key and value maps once (one tcgen05 product over all heads), and a pair costs dim + rot + v_dim = 320.
// 2,048 tokens, 16 heads: 362 us on the rows, 93 us here and 16 for the rows' copy and the maps.
//
//   latent_rows: the cached rows that the step's tokens see (whole contexts, or from the window's first key on), one request after the
//     other, out of the pages
//   latent_heads: one head x 64 tokens of one request a CTA of 4 warps x 16 rows, mma.sync m16n8k16 with float32 sums, keys and values in
//     tiles of 64 through two stages of 16-byte asynchronous copies: a key is its head's `dim` columns of the mapped rows
//     and the row's rotated part, which all heads share.  Rows padded by 8 elements, so that ldmatrix is free of bank
//     conflicts.  Softmax in float32 in units of log2(e); sinks and a gate a head as in attention_latent_mma.cu.
#include "common.cuh"
#include "mma_utils.cuh"
#include <math.h>

namespace {
constexpr int WARPS = 4, THREADS = WARPS * 32;
constexpr int BM = 64, BN = 64;
static_assert(BM == RLIS_PREFILL_TILE, "the host's tile list is cut for another tile size");
constexpr float LOG2E = 1.4426950408889634f;

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// A request's first key that a token of the step sees (the one before it by `window` - 1 keys, or key 0).
__device__ __forceinline__ int first_formed(int ctx, int q_len, int window) { return window > 0 ? max(0, ctx - q_len - window + 1) : 0; }

// The i-th key that the step sees, requests one after the other: its latent to lat[i], its rotated part to rot[i]; a warp a row,
// 16 bytes a lane.
__global__ __launch_bounds__(256) void latent_rows_kernel(const uint4* __restrict__ cache, uint4* __restrict__ lat, uint4* __restrict__ rot,
                                                          const int* __restrict__ cu_seqlens, const int* __restrict__ ctx_lens,
                                                          const int* __restrict__ block_tables, int max_blocks, int n_seqs, int page_size, int lat_vecs, int rot_vecs,
                                                          int window, int total) {
    pdl_wait();
    const int i = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (i < total) {
        int key = i, b = 0, lo, n;
        for (;; key -= n, ++b) {
            const int ctx = ctx_lens[b];
            lo = first_formed(ctx, cu_seqlens[b + 1] - cu_seqlens[b], window);
            n = ctx - lo;
            if (key < n || b == n_seqs - 1) break;
        }
        const int page = key < n ? block_tables[(size_t)b * max_blocks + (lo + key) / page_size] : -1;
        const int vecs = lat_vecs + rot_vecs;
        const uint4* src = cache + ((size_t)(page < 0 ? 0 : page) * page_size + (lo + key) % page_size) * vecs;
        for (int v = lane; v < vecs; v += 32) {
            const uint4 x = page < 0 ? make_uint4(0u, 0u, 0u, 0u) : src[v];
            if (v < lat_vecs) lat[(size_t)i * lat_vecs + v] = x;
            else rot[(size_t)i * rot_vecs + v - lat_vecs] = x;
        }
    }
    pdl_trigger();
}

struct Args {
    const bf16* q;              // [T, nh * (DIM + ROT)], q_stride apart: the plain parts are read here
    long long q_stride;
    const bf16* q_rot;          // [T, nh * ROT]: the rotated parts
    const bf16* kv;             // [keys that the step sees, nh * DIM | nh * DV]
    const bf16* rot;            // [keys that the step sees, ROT]
    bf16* out;                  // [T, nh * DV]
    const float* sinks;
    const int* tiles;
    const int* cu_seqlens;
    const int* ctx_lens;
    int nh;
    float scale;
    int window;
    const bf16* gate;
    long long gate_stride;
};

template <int DIM, int ROT, int DV>
__global__ __launch_bounds__(THREADS, 2) void latent_heads_kernel(const Args p) {
    constexpr int D = DIM + ROT, SK = D + 8, SV = DV + 8, STAGE = BN * (SK + SV);
    constexpr int KS = D / 16, ND = DV / 8;
    pdl_wait();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    bf16* sbase = reinterpret_cast<bf16*>(smem_raw);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
    const int b = p.tiles[2 * blockIdx.y], t0 = p.tiles[2 * blockIdx.y + 1], head = blockIdx.x, nh = p.nh;
    const int q_start = p.cu_seqlens[b], q_len = p.cu_seqlens[b + 1] - q_start, start_pos = p.ctx_lens[b] - q_len;
    long long key_base = -first_formed(p.ctx_lens[b], q_len, p.window);          // where the request's key 0 would lie
    for (int o = 0; o < b; ++o) key_base += p.ctx_lens[o] - first_formed(p.ctx_lens[o], p.cu_seqlens[o + 1] - p.cu_seqlens[o], p.window);

    const int r0 = warp * 16 + g, ti0 = t0 + r0, ti1 = ti0 + 8;       // this lane's two rows of the tile
    const bool rv0 = ti0 < q_len, rv1 = ti1 < q_len;
    const int pos0 = start_pos + ti0, pos1 = start_pos + ti1;
    const int lo0 = p.window > 0 ? max(0, pos0 - p.window + 1) : 0, lo1 = p.window > 0 ? max(0, pos1 - p.window + 1) : 0;
    uint32_t qa[KS][4];
    {
        const size_t t_0 = q_start + (rv0 ? ti0 : 0), t_1 = q_start + (rv1 ? ti1 : 0);
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) {
            const bool plain = ks * 16 < DIM;
            const bf16* q0 = plain ? p.q + t_0 * p.q_stride + head * D + ks * 16 : p.q_rot + (t_0 * nh + head) * ROT + ks * 16 - DIM;
            const bf16* q1 = plain ? p.q + t_1 * p.q_stride + head * D + ks * 16 : p.q_rot + (t_1 * nh + head) * ROT + ks * 16 - DIM;
            qa[ks][0] = rv0 ? *reinterpret_cast<const uint32_t*>(q0 + 2 * c) : 0u;
            qa[ks][1] = rv1 ? *reinterpret_cast<const uint32_t*>(q1 + 2 * c) : 0u;
            qa[ks][2] = rv0 ? *reinterpret_cast<const uint32_t*>(q0 + 2 * c + 8) : 0u;
            qa[ks][3] = rv1 ? *reinterpret_cast<const uint32_t*>(q1 + 2 * c + 8) : 0u;
        }
    }
    const int k_hi = start_pos + min(t0 + BM, q_len);                                  // exclusive
    const int k_lo = p.window > 0 ? max(0, start_pos + t0 - p.window + 1) : 0;
    const int kt0 = k_lo / BN, kt1 = (k_hi + BN - 1) / BN;
    const long long kv_row = (long long)nh * (DIM + DV);
    const bf16* kbase = p.kv + head * DIM;
    const bf16* vbase = p.kv + (size_t)nh * DIM + head * DV;

    auto issue = [&](int kt, int stage) {
        bf16* ks_ = sbase + stage * STAGE;
        bf16* vs_ = ks_ + BN * SK;
        auto copy = [&](bf16* dst, int pitch, const bf16* src, long long src_row, int pieces) {
#pragma unroll
            for (int i = 0; i < BN * pieces / THREADS; ++i) {
                const int idx = threadIdx.x + i * THREADS, kin = idx / pieces, c16 = idx % pieces * 8, key = kt * BN + kin;
                const bool valid = key < k_hi && key >= k_lo;
                cp_async16(dst + kin * pitch + c16, src + (key_base + (valid ? key : k_lo)) * src_row + c16, valid);
            }
        };
        copy(ks_, SK, kbase, kv_row, DIM / 8);
        copy(ks_ + DIM, SK, p.rot, ROT, ROT / 8);
        copy(vs_, SV, vbase, kv_row, DV / 8);
        cp_async_commit();
    };

    const float scale_log2 = p.scale * LOG2E;
    float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
    float oacc[ND][4];
#pragma unroll
    for (int nd = 0; nd < ND; ++nd)
#pragma unroll
        for (int e = 0; e < 4; ++e) oacc[nd][e] = 0.f;

    int stage = 0;
    if (kt0 < kt1) issue(kt0, 0);
    for (int kt = kt0; kt < kt1; ++kt) {
        if (kt + 1 < kt1) {
            issue(kt + 1, stage ^ 1);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
        const bf16* ks_ = sbase + stage * STAGE;
        const bf16* vs_ = ks_ + BN * SK;
        float sacc[8][4];
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
#pragma unroll
            for (int e = 0; e < 4; ++e) sacc[nt][e] = 0.f;
#pragma unroll
            for (int ks2 = 0; ks2 < KS / 2; ++ks2) {
                uint32_t kb[4];
                ldmatrix_x4(kb, ks_ + (nt * 8 + (lane & 7)) * SK + ks2 * 32 + (lane >> 3) * 8);
                mma_bf16_16816(sacc[nt], qa[2 * ks2], kb[0], kb[1]);
                mma_bf16_16816(sacc[nt], qa[2 * ks2 + 1], kb[2], kb[3]);
            }
        }
        // (most tiles of a long prompt: every key is seen by every row)
        const bool edge = (kt + 1) * BN - 1 > start_pos + t0 + warp * 16 || p.window > 0;
        float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
        for (int nt = 0; nt < 8; ++nt)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                float s0 = sacc[nt][e] * scale_log2, s1 = sacc[nt][2 + e] * scale_log2;
                if (edge) {
                    const int key = kt * BN + nt * 8 + 2 * c + e;
                    if (!(key <= pos0 && key >= lo0)) s0 = -INFINITY;
                    if (!(key <= pos1 && key >= lo1)) s1 = -INFINITY;
                }
                sacc[nt][e] = s0;
                sacc[nt][2 + e] = s1;
                mx0 = fmaxf(mx0, s0);
                mx1 = fmaxf(mx1, s1);
            }
        mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 1));
        mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 2));
        mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 1));
        mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 2));
        const float mn0 = fmaxf(m_run[0], mx0), mn1 = fmaxf(m_run[1], mx1);
        const float ms0 = mn0 == -INFINITY ? 0.f : mn0, ms1 = mn1 == -INFINITY ? 0.f : mn1;
        const float corr0 = ex2(m_run[0] - ms0), corr1 = ex2(m_run[1] - ms1);
        // the weights as the value product takes them, rounded to bfloat16; numerator and denominator see the same rounding
        float ls0 = 0.f, ls1 = 0.f;
        uint32_t pa[BN / 16][4];
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            const uint32_t w0 = pack_bf16(ex2(sacc[nt][0] - ms0), ex2(sacc[nt][1] - ms0)), w1 = pack_bf16(ex2(sacc[nt][2] - ms1), ex2(sacc[nt][3] - ms1));
            pa[nt / 2][nt % 2 * 2] = w0;
            pa[nt / 2][nt % 2 * 2 + 1] = w1;
            ls0 += __uint_as_float(w0 << 16) + __uint_as_float(w0 & 0xffff0000u);
            ls1 += __uint_as_float(w1 << 16) + __uint_as_float(w1 & 0xffff0000u);
        }
        ls0 += __shfl_xor_sync(0xffffffffu, ls0, 1);
        ls0 += __shfl_xor_sync(0xffffffffu, ls0, 2);
        ls1 += __shfl_xor_sync(0xffffffffu, ls1, 1);
        ls1 += __shfl_xor_sync(0xffffffffu, ls1, 2);
        l_run[0] = l_run[0] * corr0 + ls0;
        l_run[1] = l_run[1] * corr1 + ls1;
        m_run[0] = mn0;
        m_run[1] = mn1;
#pragma unroll
        for (int nd = 0; nd < ND; ++nd) {
            oacc[nd][0] *= corr0;
            oacc[nd][1] *= corr0;
            oacc[nd][2] *= corr1;
            oacc[nd][3] *= corr1;
        }
#pragma unroll
        for (int kk = 0; kk < BN / 16; ++kk) {
#pragma unroll
            for (int nd2 = 0; nd2 < ND / 2; ++nd2) {
                uint32_t vb[4];
                const int mat = lane >> 3;
                ldmatrix_x4_trans(vb, vs_ + (kk * 16 + (mat & 1) * 8 + (lane & 7)) * SV + (nd2 * 2 + (mat >> 1)) * 8);
                mma_bf16_16816(oacc[2 * nd2], pa[kk], vb[0], vb[1]);
                mma_bf16_16816(oacc[2 * nd2 + 1], pa[kk], vb[2], vb[3]);
            }
        }
        __syncthreads();       // everyone is done with this stage before the next copies land in it
        stage ^= 1;
    }
    if (p.sinks != nullptr) {
        // one more term of the denominator, without a key or a value (a sink far above every score gives inf, and 0)
        const float sink_l2 = p.sinks[head] * LOG2E;
        l_run[0] += ex2(sink_l2 - m_run[0]);
        l_run[1] += ex2(sink_l2 - m_run[1]);
    }
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        if (!(half ? rv1 : rv0)) continue;
        const size_t t = q_start + (half ? ti1 : ti0);
        float inv = l_run[half] > 0.f ? 1.0f / l_run[half] : 0.f;
        if (p.gate != nullptr) inv *= 1.0f / (1.0f + expf(-__bfloat162float(p.gate[t * p.gate_stride + head])));
        bf16* o = p.out + (t * nh + head) * DV;
#pragma unroll
        for (int nd = 0; nd < ND; ++nd)
            *reinterpret_cast<uint32_t*>(o + nd * 8 + 2 * c) = pack_bf16(oacc[nd][2 * half] * inv, oacc[nd][2 * half + 1] * inv);
    }
    pdl_trigger();
}
}  // namespace

extern "C" int rlis_latent_heads_takes(int dim, int rot, int v_dim, int rank) { return dim == 128 && rot == 64 && v_dim == 128 && rank > 0 && rank % 8 == 0; }

// cache [pages, page_size, rank + rot_width] -> lat [total, rank] and rot [total, rot_width] (bfloat16, both widths multiples of 8): for every request in
// turn the cached rows from the first one on that its first token of the step sees (with a window W: W - 1 keys back).
extern "C" int rlis_latent_rows(const void* cache, void* lat, void* rot, const int* cu_seqlens, const int* ctx_lens, const int* block_tables, int max_blocks,
                                int n_seqs, int page_size, int rank, int rot_width, int window, int total, cudaStream_t stream) {
    if (total <= 0 || n_seqs <= 0) return 0;
    if (rank <= 0 || rank % 8 || rot_width % 8 || page_size <= 0 ||
        ((reinterpret_cast<uintptr_t>(cache) | reinterpret_cast<uintptr_t>(lat) | reinterpret_cast<uintptr_t>(rot)) & 15))
        return RLIS_ERR_UNSUPPORTED;
    rlis_launch(latent_rows_kernel, (total + 7) / 8, 256, 0, stream, (const uint4*)cache, (uint4*)lat, (uint4*)rot, cu_seqlens, ctx_lens, block_tables, max_blocks,
                n_seqs, page_size, rank / 8, rot_width / 8, window, total);
    return RLIS_LAUNCH_CHECK();
}

// tiles: int32 [n_tiles][2] = (batch entry, first token of the tile within the entry's portion); kv [keys, nh * dim | nh * v_dim] and rot
// [keys, rot] in the order of rlis_latent_rows with the same window; gate (null: none): logits, head h of token t at gate[t * gate_stride + h].
extern "C" int rlis_attention_latent_heads(const void* q, long long q_stride, const void* q_rot, const void* kv, const void* rot_keys, void* out,
                                           const float* sinks, const int* tiles, int n_tiles, const int* cu_seqlens, const int* ctx_lens, int nh, int dim,
                                           int rot, int v_dim, int rank, float scale, int window, const void* gate, long long gate_stride, cudaStream_t stream) {
    if (n_tiles <= 0) return 0;
    if (!rlis_latent_heads_takes(dim, rot, v_dim, rank) || nh <= 0 || n_tiles > 65535 || q_stride % 2 || (reinterpret_cast<uintptr_t>(q) & 3) ||
        ((reinterpret_cast<uintptr_t>(kv) | reinterpret_cast<uintptr_t>(rot_keys)) & 15))
        return RLIS_ERR_UNSUPPORTED;
    constexpr int DIM = 128, ROT = 64, DV = 128, smem = 2 * BN * (DIM + ROT + 8 + DV + 8) * 2;
    const cudaError_t e = cudaFuncSetAttribute(latent_heads_kernel<DIM, ROT, DV>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    const Args p = {(const bf16*)q, q_stride, (const bf16*)q_rot, (const bf16*)kv, (const bf16*)rot_keys, (bf16*)out, sinks, tiles, cu_seqlens, ctx_lens,
                    nh, scale, window, (const bf16*)gate, gate_stride};
    rlis_launch(latent_heads_kernel<DIM, ROT, DV>, dim3(nh, n_tiles), THREADS, smem, stream, p);
    return RLIS_LAUNCH_CHECK();
}
