// Temperature sampling with top-k and/or top-p (nucleus) filtering on the device, one CTA per row
// of float32 logits, so that such rows no longer send their logits (half a megabyte at 128 k
// vocabulary) to the host.  The reference filters on the host (crates/engine/src/sampler.rs:116-221:
// weights exp((l - max) / T), the k highest logits, the shortest descending prefix whose share of
// the mass reaches top_p, an inverse-CDF draw); the rule is the same here, arranged so that no
// sort is needed and every sum is exact:
//   * weights are fixed-point integers, w = floor(exp((l - max) / T) * 2^40), added with integer
//     atomics, so sums do not depend on the order of addition and a draw is reproducible; a NaN counts
//     as -inf, infinite logits share the mass;
//   * the k-th highest logit, and then the nucleus threshold (the largest value t with
//     mass{l >= t} >= top_p * mass), are found by a radix search over the order-preserving 32-bit
//     image of the floats: four passes of 8 bits, a 256-bin histogram each (counts for top-k,
//     masses for top-p);
//   * the token is drawn from the kept set by inverse CDF in vocabulary order with a 53-bit
//     uniform that the host derives from (seed, position): r = floor(u * kept mass), the first token
//     whose running mass exceeds r.
// Of logits equal to a threshold the lowest token ids are kept, as the reference's ordering has it.
// params[r] = (bits of 1/T, top_k, bits of top_p, low and high word of the 53-bit uniform).
#include "common.cuh"
#include "mma_utils.cuh"
#include <math.h>

namespace {
constexpr int FT = 1024;
typedef unsigned long long u64;

// Every bit flipped below zero, the sign alone otherwise.  A NaN of either sign counts as -inf: it pushes no token out of a top-k
// set and weighs nothing.
__device__ __forceinline__ uint32_t order_key(float f) {
    const uint32_t u = __float_as_uint(f);
    if ((u & 0x7fffffffu) > 0x7f800000u) return 0x007fffffu;
    return u ^ ((uint32_t)((int)u >> 31) | 0x80000000u);
}
__device__ __forceinline__ float key_value(uint32_t key) {
    return __uint_as_float((key & 0x80000000u) ? (key & 0x7fffffffu) : ~key);
}
// `mx` is not -inf.  (inf - inf is a NaN, of which and of 1 the smaller is 1: infinite logits share the mass.)
__device__ __forceinline__ u64 fixed_weight(uint32_t key, float mx, float inv_t) {
    const float w = fminf(expf((key_value(key) - mx) * inv_t), 1.0f);           // in [0, 1]
    return (u64)(w * 1099511627776.0f);                                          // * 2^40
}
__device__ __forceinline__ u64 block_sum_u64(u64 v, u64* scratch) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    if (warp == 0) {
        u64 s = lane < FT / 32 ? scratch[lane] : 0ull;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) scratch[32] = s;
    }
    __syncthreads();
    const u64 r = scratch[32];
    __syncthreads();
    return r;
}

// Over the row: how many keys exceed `key0`, how many equal it, and the mass of those that exceed it.
__device__ __forceinline__ void key_stats(const float* row, int vocab, uint32_t key0, float mx, float inv_t,
                                          u64* scratch, u64& n_above, u64& n_ties, u64& mass_above) {
    u64 a = 0ull, t = 0ull, m = 0ull;
    for (int v = threadIdx.x; v < vocab; v += FT) {
        const uint32_t key = order_key(row[v]);
        if (key > key0) { ++a; m += fixed_weight(key, mx, inv_t); }
        else if (key == key0) ++t;
    }
    n_above = block_sum_u64(a, scratch);
    n_ties = block_sum_u64(t, scratch);
    mass_above = block_sum_u64(m, scratch);
}

__global__ __launch_bounds__(FT) void sample_filtered_kernel(const float* __restrict__ logits,
                                                             const uint32_t* __restrict__ params,
                                                             int* __restrict__ out, int vocab,
                                                             long long row_stride) {
    pdl_wait();
    __shared__ u64 hist[256];
    __shared__ u64 scratch[33];
    __shared__ u64 scan_a[FT / 32], scan_b[FT / 32];
    __shared__ float s_max[FT / 32];
    __shared__ uint32_t s_prefix;
    __shared__ u64 s_above;
    __shared__ int s_owner;
    const int r = blockIdx.x;
    const float* row = logits + (size_t)r * row_stride;
    const float inv_t = __uint_as_float(params[5 * r]);
    const int top_k = (int)params[5 * r + 1];
    const float top_p = __uint_as_float(params[5 * r + 2]);
    const u64 u53 = (u64)params[5 * r + 3] | ((u64)params[5 * r + 4] << 32);
    const bool use_k = top_k > 0 && top_k < vocab;
    const bool use_p = top_p < 1.0f;

    // the row's maximum
    float mx = -INFINITY;
    for (int v = threadIdx.x; v < vocab; v += FT) mx = fmaxf(mx, row[v]);
    mx = warp_max(mx);
    if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = mx;
    __syncthreads();
    mx = s_max[0];
    for (int i = 1; i < FT / 32; ++i) mx = fmaxf(mx, s_max[i]);
    __syncthreads();
    if (mx == -INFINITY) mx = 0.f;          // nothing to draw: no token weighs anything

    // top-k: the k-th highest key by radix search on counts
    uint32_t kth = 0u;
    if (use_k) {
        uint32_t prefix = 0u;
        u64 k_rem = (u64)top_k;
        for (int pass = 0; pass < 4; ++pass) {
            const int shift = 24 - 8 * pass;
            for (int i = threadIdx.x; i < 256; i += FT) hist[i] = 0ull;
            __syncthreads();
            for (int v = threadIdx.x; v < vocab; v += FT) {
                const uint32_t key = order_key(row[v]);
                if (pass == 0 || (key >> (shift + 8)) == (prefix >> (shift + 8)))
                    atomicAdd(&hist[(key >> shift) & 255u], 1ull);
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                u64 cum = 0ull;
                int b = 255;
                for (; b > 0; --b) {
                    if (cum + hist[b] >= k_rem) break;
                    cum += hist[b];
                }
                s_prefix = prefix | ((uint32_t)b << shift);
                s_above = cum;
            }
            __syncthreads();
            prefix = s_prefix;
            k_rem -= s_above;
            __syncthreads();
        }
        kth = prefix;
    }
    // Of the logits equal to the k-th one only as many as top_k still has room for are kept, lowest
    // ids first (crates/engine/src/sampler.rs:182-195).
    u64 n_above_k, n_ties_k, mass_above_k;
    key_stats(row, vocab, kth, mx, inv_t, scratch, n_above_k, n_ties_k, mass_above_k);
    const u64 keep_k = use_k ? (u64)top_k - n_above_k : n_ties_k;
    const u64 w_k = fixed_weight(kth, mx, inv_t);
    const u64 mass = mass_above_k + keep_k * w_k;        // of the top-k set (or of everything)

    // top-p: the largest threshold whose upper mass reaches top_p * mass, by radix search on masses
    uint32_t thr = kth;
    u64 tie_keep = keep_k;
    if (use_p) {
        const u64 target = (u64)((double)top_p * (double)mass);
        uint32_t prefix = 0u;
        u64 above = 0ull;                     // mass of keys above the bins chosen so far
        for (int pass = 0; pass < 4; ++pass) {
            const int shift = 24 - 8 * pass;
            for (int i = threadIdx.x; i < 256; i += FT) hist[i] = 0ull;
            __syncthreads();
            for (int v = threadIdx.x; v < vocab; v += FT) {
                const uint32_t key = order_key(row[v]);
                if (key >= kth && (pass == 0 || (key >> (shift + 8)) == (prefix >> (shift + 8))))
                    atomicAdd(&hist[(key >> shift) & 255u], fixed_weight(key, mx, inv_t));
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                u64 cum = above;
                int b = 255;
                for (; b > 0; --b) {
                    if (cum + hist[b] >= target && hist[b] > 0ull) break;
                    cum += hist[b];
                }
                s_prefix = prefix | ((uint32_t)b << shift);
                s_above = cum;
            }
            __syncthreads();
            prefix = s_prefix;
            above = s_above;
            __syncthreads();
        }
        thr = prefix > kth ? prefix : kth;
        // of the logits equal to the threshold, the lowest ids are kept until the mass is reached
        // (the crossing token included; sampler.rs:200-209)
        u64 n_above, n_ties, mass_above;
        key_stats(row, vocab, thr, mx, inv_t, scratch, n_above, n_ties, mass_above);
        const u64 w_t = fixed_weight(thr, mx, inv_t);
        u64 need = 1ull;
        if (target > mass_above && w_t > 0ull) need = (target - mass_above + w_t - 1ull) / w_t;
        if (need < 1ull) need = 1ull;
        const u64 room = thr == kth ? keep_k : n_ties;
        tie_keep = need < room ? need : room;
    }

    // inverse CDF over the kept set in vocabulary order: a contiguous piece of the row per thread
    const int per = (vocab + FT - 1) / FT;
    const int v0 = min(threadIdx.x * per, vocab), v1 = min(v0 + per, vocab);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // rank of this piece's first tie among all logits equal to the threshold
    u64 my_ties = 0ull;
    for (int v = v0; v < v1; ++v) my_ties += order_key(row[v]) == thr ? 1ull : 0ull;
    u64 incl_t = my_ties;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const u64 n = __shfl_up_sync(0xffffffffu, incl_t, o);
        if (lane >= o) incl_t += n;
    }
    if (lane == 31) scan_a[warp] = incl_t;
    __syncthreads();
    u64 tie_rank = incl_t - my_ties;
    for (int i = 0; i < warp; ++i) tie_rank += scan_a[i];
    // kept mass of this piece
    u64 mine = 0ull, rank = tie_rank;
    for (int v = v0; v < v1; ++v) {
        const uint32_t key = order_key(row[v]);
        if (key > thr || (key == thr && rank++ < tie_keep)) mine += fixed_weight(key, mx, inv_t);
    }
    u64 incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const u64 n = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += n;
    }
    if (lane == 31) scan_b[warp] = incl;
    if (threadIdx.x == 0) s_owner = -1;
    __syncthreads();
    u64 warp_base = 0ull, kept = 0ull;
    for (int i = 0; i < FT / 32; ++i) {
        if (i < warp) warp_base += scan_b[i];
        kept += scan_b[i];
    }
    const u64 before = warp_base + incl - mine;
    // r = floor(u * kept), u = u53 / 2^53
    const u64 target_r = __umul64hi(u53 << 11, kept);
    if (mine > 0ull && target_r >= before && target_r < before + mine) s_owner = threadIdx.x;
    __syncthreads();
    if ((int)threadIdx.x == s_owner) {
        u64 cum = before, rk = tie_rank;
        int pick = v1 - 1;
        for (int v = v0; v < v1; ++v) {
            const uint32_t key = order_key(row[v]);
            if (key > thr || (key == thr && rk++ < tie_keep)) {
                cum += fixed_weight(key, mx, inv_t);
                if (cum > target_r) { pick = v; break; }
            }
        }
        out[r] = pick;
    }
    if (s_owner < 0 && threadIdx.x == 0) out[r] = 0;   // nothing kept (a row of NaNs or -inf): id 0, as the greedy path
    pdl_trigger();   // the next kernel of the stream may start its launch
}

int g_filtered_cluster = 1;      // 0: the one-CTA kernel for every vocabulary (tests of that kernel)

// ------------------------------------------------------------------------------------------------
// The same rule with a thread-block cluster per row: CC CTAs of 512 threads hold the row's order keys in registers (thread
// t of CTA c: E consecutive token ids, so that CTA order and thread order are vocabulary order), every pass
// works on registers, histograms and sums of the CTAs meet through distributed shared memory, and every CTA draws the same
// conclusions from the same totals.  Same integers, same token as the one-CTA kernel above, which stays for
// vocabularies too large for it.
//
// A threshold is found by narrowing an interval of keys in histograms of 1,024 bins, counted from the top.  The first one
// takes bins of 2^17 keys down from the row's highest key: 64 bins an octave of the logits' values over sixteen octaves,
// so logits that crowd into a few octaves still spread over hundreds of bins (with 8 bits of the key a pass they met in half a dozen, and
// the adds in shared memory queued up).  What lies further down is left out and only looked at if the threshold is
// not above it.  The tokens of the bin that holds the threshold, a hundred or two, are then put in one list and
// compared each with each; only where there are more than 256 (ties, above all) the bins narrow further, to 2^7 keys and to
// one.  A top-k set of up to 256 goes to the list at once when top-p narrows it.  Masses are added as
// three 32-bit numbers of 14, 14 and 13 bits of the weight: a CTA's 16,384 tokens cannot overflow them, and shared memory adds
// 32 bits natively.  The first histogram of masses is filled in the pass that adds up the whole mass, and
// weights are made again from the keys where they are needed, so that a thread stays within 64 registers and two CTAs
// share an SM.  64 rows of 128,256 logits with top-p, top-k or both: 410 us with 8-bit passes, 103 us.
constexpr int CT = 512;

__device__ __forceinline__ u64 ld_dsmem_u64(const u64* local, uint32_t rank) {
    uint32_t remote;
    u64 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(local)), "r"(rank));
    asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(v) : "r"(remote) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t ld_dsmem_u32(const uint32_t* local, uint32_t rank) {
    uint32_t remote, v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(local)), "r"(rank));
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(remote) : "memory");
    return v;
}

// The values at one shared-memory offset in all CTAs of the cluster, added in rank order.
__device__ __forceinline__ u64 cluster_total_u64(const u64* local, uint32_t cc) {
    u64 t = 0ull;
    for (uint32_t c = 0; c < cc; ++c) t += ld_dsmem_u64(local, c);
    return t;
}
constexpr int BINS = 1024, TOP_SHIFT = 17;
constexpr uint32_t LIST = 256;       // tokens that are compared one with the other, a thread each (all pairs: 4 us; a level of bins takes 5)

struct ClusterShared {
    uint32_t hist[3][3][BINS];   // a level's counts, or its masses in three parts; three levels in turn: one is filled, the one before it
                                 // may still be read by other CTAs, the one after it is emptied
    u64 xch[8];                  // a CTA's sum of a phase, read by the whole cluster
    float xmax;
    uint32_t xkey;
    float fmax_of[CT / 32];
    uint32_t kmax_of[CT / 32];
    u64 scan[CT / 32];
    int best;
    u64 above, inside;
    uint32_t n_list, best_key;
    uint32_t list[LIST], all_keys[LIST];
    u64 all_values[LIST];
};

__device__ __forceinline__ uint2 ld_dsmem_2u32(const uint32_t* local, uint32_t rank) {
    uint32_t remote;
    uint2 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(local)), "r"(rank));
    asm volatile("ld.shared::cluster.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(remote) : "memory");
    return v;
}

// This thread's share of a sum over the CTA, inclusive of the threads before it in order, and the CTA's sum.
__device__ __forceinline__ u64 cta_prefix_u64(u64 mine, u64* scan, u64& total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    u64 incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const u64 n = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += n;
    }
    if (lane == 31) scan[warp] = incl;
    __syncthreads();
    u64 before = 0ull;
    total = 0ull;
#pragma unroll
    for (int i = 0; i < CT / 32; ++i) {
        const u64 w = scan[i];
        if (i < warp) before += w;
        total += w;
    }
    __syncthreads();
    return before + incl;
}

template <int E>
__global__ __launch_bounds__(CT, 2) void sample_filtered_cluster_kernel(const float* __restrict__ logits,
                                                                        const uint32_t* __restrict__ params,
                                                                        int* __restrict__ out, int vocab,
                                                                        long long row_stride) {
    pdl_wait();
    __shared__ ClusterShared sh;
    const uint32_t rank = blockIdx.x, cc = gridDim.x;
    const int r = blockIdx.y;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float* row = logits + (size_t)r * row_stride;
    const float inv_t = __uint_as_float(params[5 * r]);
    const int top_k = (int)params[5 * r + 1];
    const float top_p = __uint_as_float(params[5 * r + 2]);
    const u64 u53 = (u64)params[5 * r + 3] | ((u64)params[5 * r + 4] << 32);
    const bool use_k = top_k > 0 && top_k < vocab;
    const bool use_p = top_p < 1.0f;

    // this thread's E consecutive tokens; those past the vocabulary take part in nothing
    const int v0 = ((int)rank * CT + tid) * E;
    const int n_mine = max(0, min(E, vocab - v0));
    uint32_t key[E];
    float mx = -INFINITY;
    uint32_t top_key = 0u;
    if (((reinterpret_cast<uintptr_t>(row) & 15) == 0) && n_mine == E) {
#pragma unroll
        for (int i = 0; i < E; i += 4) {
            const float4 x = *reinterpret_cast<const float4*>(row + v0 + i);
            mx = fmaxf(fmaxf(mx, fmaxf(x.x, x.y)), fmaxf(x.z, x.w));
            key[i] = order_key(x.x); key[i + 1] = order_key(x.y); key[i + 2] = order_key(x.z); key[i + 3] = order_key(x.w);
        }
    } else {
#pragma unroll
        for (int i = 0; i < E; ++i) {
            const float l = i < n_mine ? row[v0 + i] : -INFINITY;
            mx = fmaxf(mx, l);
            key[i] = i < n_mine ? order_key(l) : 0u;
        }
    }
#pragma unroll
    for (int i = 0; i < E; ++i) top_key = max(top_key, key[i]);

    // the row's maximum, and its highest key
    mx = warp_max(mx);
    top_key = __reduce_max_sync(0xffffffffu, top_key);
    if (lane == 0) { sh.fmax_of[warp] = mx; sh.kmax_of[warp] = top_key; }
    for (int i = tid; i < 3 * BINS; i += CT) sh.hist[0][0][i] = 0u;
    __syncthreads();
    if (tid == 0) {
        for (int i = 1; i < CT / 32; ++i) { mx = fmaxf(mx, sh.fmax_of[i]); top_key = max(top_key, sh.kmax_of[i]); }
        sh.xmax = mx;
        sh.xkey = top_key;
    }
    cluster_sync_all();
    for (uint32_t c = 0; c < cc; ++c) {
        mx = fmaxf(mx, ld_dsmem(&sh.xmax, c));
        top_key = max(top_key, ld_dsmem_u32(&sh.xkey, c));
    }
    if (mx == -INFINITY) mx = 0.f;              // nothing to draw: no token weighs anything
    auto weight = [&](int i) -> u64 { return fixed_weight(key[i], mx, inv_t); };

    int buf = 0, phase = 0;
    // The highest key such that the counts (`masses` false) or masses of the keys from it upwards reach `need_of(sum)`, of the
    // tokens whose key is at least `lower` (`sum`: the mass of all those above `lower`, 0 for counts).  `above`: what lies
    // above it, `inside`: what equals it.  `known`: how many tokens there are at `lower` and above, if known.
    auto select = [&](auto need_of, bool masses, uint32_t lower, u64 known, u64& above, u64& inside) -> uint32_t {
        uint32_t hi = top_key, lo = lower;         // the threshold lies in lo .. hi
        int shift = TOP_SHIFT;
        u64 need = 0ull;
        above = 0ull;
        bool first = true;                         // `need` is not known yet
        for (bool try_list = known <= LIST;;) {
            if (try_list) {
                // few tokens may be left: all of them in one list, where each is compared with each
                if (tid == 0) sh.n_list = 0u;
                __syncthreads();
#pragma unroll
                for (int i = 0; i < E; ++i) {
                    if (key[i] >= lo && key[i] <= hi && i < n_mine) {
                        const uint32_t at = atomicAdd(&sh.n_list, 1u);
                        if (at < LIST) sh.list[at] = key[i];
                    }
                }
                if (tid == 0) sh.best_key = 0u;
                cluster_sync_all();
                uint32_t n = 0u, mine = 0u;
                for (uint32_t c = 0; c < cc; ++c) {
                    const uint32_t nc = ld_dsmem_u32(&sh.n_list, c);
                    if (n <= LIST && nc <= LIST && tid >= n && tid < n + nc) mine = ld_dsmem_u32(&sh.list[tid - n], c);
                    n = min(n + nc, LIST + 1u);
                }
                if (n <= LIST) {
                    const u64 v = tid < n ? (masses ? fixed_weight(mine, mx, inv_t) : 1ull) : 0ull;
                    if (tid < n) { sh.all_keys[tid] = mine; sh.all_values[tid] = v; }
                    __syncthreads();
                    u64 higher = 0ull, equal = 0ull;
                    for (uint32_t j = 0; j < (warp * 32 < (int)n ? n : 0u); ++j) {
                        const uint32_t k = sh.all_keys[j];
                        const u64 w = sh.all_values[j];
                        if (k > mine) higher += w;
                        if (k == mine) equal += w;
                    }
                    if (first) {
                        u64 sum;
                        cta_prefix_u64(mine > lower ? v : 0ull, sh.scan, sum);
                        need = need_of(sum);
                    }
                    const bool here = tid < n && equal > 0ull && above + higher + equal >= need;
                    if (here) atomicMax(&sh.best_key, mine);
                    __syncthreads();
                    const uint32_t best = sh.best_key;
                    if (here && mine == best) { sh.above = above + higher; sh.inside = equal; }     // (the same of all that are equal)
                    if (tid == 0 && best == 0u) sh.inside = 0ull;                                       // nothing reaches the need
                    __syncthreads();
                    if (best != 0u) above = sh.above;
                    inside = sh.inside;
                    cluster_sync_all();             // (the lists have been read before another one is made)
                    return best != 0u ? best : lower;
                }
                cluster_sync_all();
            }
            uint32_t (*hist)[BINS] = sh.hist[buf];
            u64 sum = 0ull;
#pragma unroll
            for (int i = 0; i < E; ++i) {
                const uint32_t bin = (hi - key[i]) >> shift;
                const bool in = key[i] <= hi && key[i] >= lo && bin < BINS && i < n_mine;
                if (!masses) {
                    if (in) atomicAdd(&hist[0][bin], 1u);
                } else if (in || (first && key[i] >= lower && i < n_mine)) {
                    const u64 w = weight(i);
                    if (in && w != 0ull) {
                        atomicAdd(&hist[0][bin], (uint32_t)w & 0x3FFFu);
                        atomicAdd(&hist[1][bin], (uint32_t)(w >> 14) & 0x3FFFu);
                        atomicAdd(&hist[2][bin], (uint32_t)(w >> 28));
                    }
                    if (key[i] > lower || lower == 0u) sum += w;
                }
            }
            const int next = buf == 2 ? 0 : buf + 1;
            for (int i = tid; i < 3 * BINS; i += CT) sh.hist[next][0][i] = 0u;      // (read last before the cluster barrier before this one)
            if (masses && first) {
                u64 own_sum;
                cta_prefix_u64(sum, sh.scan, own_sum);
                if (tid == 0) sh.xch[phase] = own_sum;
            }
            if (tid == 0) sh.best = BINS;
            cluster_sync_all();
            // bins 2 tid and 2 tid + 1 of all CTAs
            u64 t0 = 0ull, t1 = 0ull;
            for (uint32_t c = 0; c < cc; ++c) {
                const uint2 a = ld_dsmem_2u32(&hist[0][2 * tid], c);
                t0 += a.x;
                t1 += a.y;
                if (masses) {
                    const uint2 b = ld_dsmem_2u32(&hist[1][2 * tid], c), d = ld_dsmem_2u32(&hist[2][2 * tid], c);
                    t0 += ((u64)b.x << 14) + ((u64)d.x << 28);
                    t1 += ((u64)b.y << 14) + ((u64)d.y << 28);
                }
            }
            if (first) {
                need = need_of(masses ? cluster_total_u64(&sh.xch[phase], cc) : 0ull);
                phase += masses ? 1 : 0;
                first = false;
            }
            u64 all;
            const u64 incl = above + cta_prefix_u64(t0 + t1, sh.scan, all);      // sum down to the second of this thread's bins
            if (t0 > 0ull && incl - t1 >= need) atomicMin(&sh.best, 2 * tid);
            else if (t1 > 0ull && incl >= need) atomicMin(&sh.best, 2 * tid + 1);
            __syncthreads();
            const int best = sh.best;
            if (best < BINS && tid == best >> 1) {
                sh.above = (best & 1) ? incl - t1 : incl - t1 - t0;
                sh.inside = (best & 1) ? t1 : t0;
            }
            __syncthreads();
            buf = next;
            if (best < BINS) {
                above = sh.above;
                hi -= (uint32_t)best << shift;
                const uint32_t wide = (1u << shift) - 1u;
                lo = max(lo, hi > wide ? hi - wide : 0u);
                if (shift == 0) { inside = sh.inside; return hi; }
                // (counts say how many are left: thousands of equal tokens would queue up at the list's counter for nothing;
                // 64 rows of 32,000 logits in steps of one, top-k 5,000: 61 us with the attempt, 46 without)
                try_list = masses || sh.inside <= LIST;
            } else {                                // further down than the bins reach (never within an interval narrowed before)
                above += all;
                const uint32_t covered = shift >= 22 ? 0xFFFFFFFFu : ((uint32_t)BINS << shift) - 1u;
                if (hi - lo <= covered) { inside = 0ull; return lower; }      // nothing reaches the need
                hi -= covered + 1u;
                try_list = false;
            }
            shift = max(0, 22 - __clz(hi - lo | 1u));       // the next level's bins cover the interval
        }
    };

    // the top-k set: everything above `kth` and the first `keep_k` (in token order) of the logits equal to it
    uint32_t kth = 0u;
    u64 n_above_k = 0ull, n_ties_k = 0ull, keep_k = ~0ull;
    if (use_k) {
        kth = select([&](u64) { return (u64)top_k; }, false, 0u, ~0ull, n_above_k, n_ties_k);
        keep_k = (u64)top_k - n_above_k;
    }
    uint32_t thr = kth;
    u64 tie_keep = keep_k, n_ties = use_k ? n_ties_k : 0ull;
    if (use_p) {
        // the largest threshold whose upper mass reaches top_p * mass
        const u64 w_k = use_k ? fixed_weight(kth, mx, inv_t) : 0ull;
        u64 target = 0ull, above, inside;
        thr = select([&](u64 mass_above_k) {
            const u64 mass = mass_above_k + (use_k ? keep_k * w_k : 0ull);
            target = (u64)((double)top_p * (double)mass);
            return target;
        }, true, kth, use_k ? n_above_k + n_ties_k : ~0ull, above, inside);
        const u64 w_t = fixed_weight(thr, mx, inv_t);
        n_ties = thr == kth && use_k ? n_ties_k : w_t > 0ull ? inside / w_t : 0ull;
        u64 need = 1ull;
        if (target > above && w_t > 0ull) need = (target - above + w_t - 1ull) / w_t;
        const u64 room = thr == kth && use_k ? keep_k : n_ties;
        tie_keep = need < room ? need : room;
    }

    // An exclusive prefix over the vocabulary order (CTA after CTA, thread after thread) of a value
    // per thread; also the cluster's total.
    auto ordered_prefix = [&](u64 mine, u64& total) -> u64 {
        u64 cta_total;
        u64 before = cta_prefix_u64(mine, sh.scan, cta_total) - mine;
        u64* slot = &sh.xch[phase];
        ++phase;
        if (tid == 0) *slot = cta_total;
        cluster_sync_all();
        total = 0ull;
        for (uint32_t c = 0; c < cc; ++c) {
            const u64 t = ld_dsmem_u64(slot, c);
            if (c < rank) before += t;
            total += t;
        }
        return before;
    };
    // rank of this thread's first tie among all logits equal to the threshold (all of them kept: no matter)
    u64 tie_rank = 0ull;
    if (tie_keep < n_ties) {
        u64 my_ties = 0ull, all_ties;
#pragma unroll
        for (int i = 0; i < E; ++i) my_ties += (i < n_mine && key[i] == thr) ? 1ull : 0ull;
        tie_rank = ordered_prefix(my_ties, all_ties);
    } else {
        tie_keep = ~0ull;
    }
    // kept mass of this thread's tokens
    u64 mine = 0ull, rk = tie_rank;
#pragma unroll
    for (int i = 0; i < E; ++i)
        if (i < n_mine && (key[i] > thr || (key[i] == thr && rk++ < tie_keep))) mine += weight(i);
    u64 kept;
    const u64 before = ordered_prefix(mine, kept);
    const u64 target_r = __umul64hi(u53 << 11, kept);          // floor(u * kept), u = u53 / 2^53
    if (mine > 0ull && target_r >= before && target_r < before + mine) {
        u64 cum = before, rk2 = tie_rank;
        int pick = v0 + n_mine - 1;
#pragma unroll
        for (int i = 0; i < E; ++i) {
            if (i < n_mine && (key[i] > thr || (key[i] == thr && rk2++ < tie_keep))) {
                cum += weight(i);
                if (cum > target_r) { pick = v0 + i; break; }
            }
        }
        out[r] = pick;
    }
    if (kept == 0ull && rank == 0 && tid == 0) out[r] = 0;     // nothing kept (a row of NaNs or -inf): id 0, as the greedy path
    cluster_sync_all();          // nobody leaves while its shared memory may still be read
    pdl_trigger();
}

template <int E>
void launch_filtered_cluster(const float* logits, const uint32_t* params, int* out, int rows, int vocab,
                             long long row_stride, int cc, cudaStream_t stream) {
    static bool attr_done = false;
    if (!attr_done) {
        cudaFuncSetAttribute(sample_filtered_cluster_kernel<E>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        attr_done = true;
    }
    rlis_launch_cluster(sample_filtered_cluster_kernel<E>, dim3((unsigned)cc, (unsigned)rows), CT, 0, stream,
                        dim3((unsigned)cc, 1, 1), logits, params, out, vocab, row_stride);
}
}  // namespace

extern "C" int rlis_sample_filtered(const float* logits, const uint32_t* params, int* out, int rows, int vocab,
                                    long long row_stride, cudaStream_t stream) {
    if (rows <= 0) return 0;
    if (vocab <= 0) return RLIS_ERR_UNSUPPORTED;
    // a cluster of 8 (16 for the largest) CTAs of 512 threads holds the row in registers, 8 to 32
    // tokens a thread; vocabularies beyond 262,144 go to the one-CTA kernel
    const long long per8 = ((long long)vocab + 8 * CT - 1) / (8 * CT);
    if (g_filtered_cluster && per8 <= 8) launch_filtered_cluster<8>(logits, params, out, rows, vocab, row_stride, 8, stream);
    else if (g_filtered_cluster && per8 <= 16) launch_filtered_cluster<16>(logits, params, out, rows, vocab, row_stride, 8, stream);
    else if (g_filtered_cluster && per8 <= 32) launch_filtered_cluster<32>(logits, params, out, rows, vocab, row_stride, 8, stream);
    else if (g_filtered_cluster && per8 <= 64) launch_filtered_cluster<32>(logits, params, out, rows, vocab, row_stride, 16, stream);
    else rlis_launch(sample_filtered_kernel, rows, FT, 0, stream, logits, params, out, vocab, row_stride);
    return RLIS_LAUNCH_CHECK();
}

extern "C" void rlis_sample_filtered_set_cluster(int on) { g_filtered_cluster = on; }
