// True 32-bit matrix product for the float32 path: C[M, N] = A[M, K] * W[N, K]^T with FFMA on the
// CUDA cores, for rows shorter than 2,048, rows off 16-byte boundaries or less than their length apart, and batches (others: gemm_f32_split.cu).  Every output element is accumulated over k = 0..K-1 in
// that order, one fused multiply-add after the other, whichever kernel below computes it and
// whatever M, N or the tile it falls in, so a row's result does not depend on what else is in the
// batch.  Role in the reference: `x.matmul(w.t())`, crates/model/src/layers.rs:82.
#include "common.cuh"
#include "mma_utils.cuh"

namespace {

// One product, and the strides of a batch of them (blockIdx.z).
struct Product {
    const float* A;
    const float* W;
    float* C;
    int M, N, K;
    long long lda, ldw, ldc, sa, sw, sc;
};

// ------------------------------------------------------------------------------------------------
// Many rows: BM x BN outputs a CTA of 256 threads, (BM / 16) x (BN / 16) a thread, in slices of 16 of k.  Bound by the
// FMA pipes and, close behind, by reads of shared memory: 4 vector loads feed 64 FMAs, issued as 32 two-wide ones
// (fma.rn.f32x2, the same roundings; 8 % faster than 64 single ones), and the next slice's global loads are in
// registers while this one is multiplied.  A warp covers 4 x 8 threads, so that each of its loads is one pass.
// 2,048 rows, N 16384, K 2048: 2.64 ms, 52 TFLOP/s of the 74 that the FMA pipes have (6.34 ms with 4 x 4 outputs a thread
// and no prefetch).
constexpr int BK = 16, TILE_THREADS = 256;

__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

template <int BM, int BN, bool VEC>
__global__ __launch_bounds__(TILE_THREADS, BM * BN >= 128 * 128 ? 2 : 3) void sgemm_nt_kernel(const Product p) {
    constexpr int TM = BM / 16, TN = BN / 16;       // outputs a thread: (TM / 4) x (TN / 4) blocks of 4 x 4
    constexpr int LDA = BM + 4, LDW = BN + 4;
    constexpr int NA = BM * BK / 4 / TILE_THREADS, NW = BN * BK / 4 / TILE_THREADS;      // 16-byte pieces a thread loads a slice
    static_assert(TM % 4 == 0 && TN % 4 == 0 && NA >= 1 && NW >= 1, "tile");
    __shared__ __align__(16) float As[2][BK][LDA];
    __shared__ __align__(16) float Ws[2][BK][LDW];
    pdl_wait();
    const float* __restrict__ A = p.A + blockIdx.z * p.sa;
    const float* __restrict__ W = p.W + blockIdx.z * p.sw;
    float* __restrict__ C = p.C + blockIdx.z * p.sc;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tx = (warp & 1) * 8 + (lane & 7), ty = (warp >> 1) * 4 + (lane >> 3);
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;

    float4 ra[NA], rw[NW];
    auto load = [&](const float* __restrict__ X, long long ld, int row, int rows, int k) -> float4 {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row >= rows) return v;
        const float* src = X + (size_t)row * ld + k;
        if (VEC) {
            if (k < p.K) v = *reinterpret_cast<const float4*>(src);         // (K is a multiple of 4)
        } else {
            if (k < p.K) v.x = src[0];
            if (k + 1 < p.K) v.y = src[1];
            if (k + 2 < p.K) v.z = src[2];
            if (k + 3 < p.K) v.w = src[3];
        }
        return v;
    };
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < NA; ++i) {
            const int piece = tid + i * TILE_THREADS;
            ra[i] = load(A, p.lda, m0 + piece / 4, p.M, k0 + piece % 4 * 4);
        }
#pragma unroll
        for (int i = 0; i < NW; ++i) {
            const int piece = tid + i * TILE_THREADS;
            rw[i] = load(W, p.ldw, n0 + piece / 4, p.N, k0 + piece % 4 * 4);
        }
    };
    auto keep = [&](int buf) {
#pragma unroll
        for (int i = 0; i < NA; ++i) {
            const int piece = tid + i * TILE_THREADS, r = piece / 4, c = piece % 4 * 4;
            As[buf][c][r] = ra[i].x; As[buf][c + 1][r] = ra[i].y; As[buf][c + 2][r] = ra[i].z; As[buf][c + 3][r] = ra[i].w;
        }
#pragma unroll
        for (int i = 0; i < NW; ++i) {
            const int piece = tid + i * TILE_THREADS, r = piece / 4, c = piece % 4 * 4;
            Ws[buf][c][r] = rw[i].x; Ws[buf][c + 1][r] = rw[i].y; Ws[buf][c + 2][r] = rw[i].z; Ws[buf][c + 3][r] = rw[i].w;
        }
    };

    unsigned long long acc[TM][TN / 2];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0ull;

    fetch(0);
    keep(0);
    __syncthreads();
    const int slices = (p.K + BK - 1) / BK;
    for (int s = 0; s < slices; ++s) {
        const int buf = s & 1;
        if (s + 1 < slices) fetch((s + 1) * BK);
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            float a[TM];
            unsigned long long b[TN / 2];
#pragma unroll
            for (int i = 0; i < TM; i += 4)
                *reinterpret_cast<float4*>(&a[i]) = *reinterpret_cast<const float4*>(&As[buf][kk][i * 16 + ty * 4]);
#pragma unroll
            for (int j = 0; j < TN; j += 4)
                *reinterpret_cast<ulonglong2*>(&b[j / 2]) = *reinterpret_cast<const ulonglong2*>(&Ws[buf][kk][j * 16 + tx * 4]);
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const unsigned long long aa = pack2(a[i], a[i]);
#pragma unroll
                for (int j = 0; j < TN / 2; ++j) fma2(acc[i][j], aa, b[j]);
            }
        }
        if (s + 1 < slices) {
            keep(buf ^ 1);              // (read last in the slice before this one, and a barrier lies in between)
            __syncthreads();
        }
    }
    const bool wide = VEC && (p.ldc & 3) == 0 && (p.sc & 3) == 0 && (reinterpret_cast<uintptr_t>(p.C) & 15) == 0;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gm = m0 + i / 4 * 64 + ty * 4 + i % 4;
        if (gm >= p.M) continue;
        float* row = C + (size_t)gm * p.ldc;
#pragma unroll
        for (int j = 0; j < TN; j += 4) {
            const int gn = n0 + j * 16 + tx * 4;
            float v[4];
            *reinterpret_cast<ulonglong2*>(v) = *reinterpret_cast<ulonglong2*>(&acc[i][j / 2]);
            if (wide && gn + 3 < p.N) {
                *reinterpret_cast<float4*>(row + gn) = *reinterpret_cast<float4*>(v);
            } else {
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (gn + u < p.N) row[gn + u] = v[u];
            }
        }
    }
    pdl_trigger();   // the next kernel of the stream may start its launch
}

// ------------------------------------------------------------------------------------------------
// Few rows (a decode step): every weight is read once, so the bound is the memory's rate over W, and below it the
// chain of K dependent FMAs that an output is (4 cycles each).  A CTA takes FB features and ROWS rows, a thread one
// feature and RB rows.  W and the rows arrive in slices of KT of k through a ring of STAGES filled by 16-byte
// asynchronous copies whose addresses a thread keeps from slice to slice (worked out anew each time they cost more than
// the products: 83 against 39 us below); rows of a slice are KT + 4 floats apart in shared memory, so that the 16-byte reads
// of neighbouring features fall in different banks, and a row of A is read by all features of a warp at once.
// 8 rows, K 8192, N 2048: 38.6 us (1.42 ms in 64 x 64 tiles); K 2048, N 16384: 43 us (391).
template <int FB, int ROWS, int RB> struct FewRows {
    static constexpr int THREADS = FB * ROWS / RB > 128 ? FB * ROWS / RB : 128;
};

template <int FB, int ROWS, int RB, int KT, int STAGES>
__global__ __launch_bounds__((FewRows<FB, ROWS, RB>::THREADS)) void sgemm_few_rows_kernel(const Product p) {
    constexpr int THREADS = FewRows<FB, ROWS, RB>::THREADS, LD = KT + 4, PIECES = KT / 4;
    constexpr int STEP = THREADS / PIECES;                           // rows of a slice between two pieces of a thread
    constexpr int NP = (FB + ROWS + STEP - 1) / STEP;                // 16-byte pieces a thread copies a slice
    constexpr int STAGE_FLOATS = (FB + ROWS) * LD;
    static_assert(THREADS % PIECES == 0 && ROWS % RB == 0, "few rows");
    extern __shared__ __align__(16) float ring[];
    pdl_wait();
    const int tid = threadIdx.x, n0 = blockIdx.x * FB, row0 = blockIdx.y * ROWS;
    const float* __restrict__ A = p.A + blockIdx.z * p.sa;
    const float* __restrict__ W = p.W + blockIdx.z * p.sw;
    float* __restrict__ C = p.C + blockIdx.z * p.sc;
    const int slices = (p.K + KT - 1) / KT;

    // this thread's pieces: the same 16 bytes of every STEP-th row (rows beyond the last are read as the last one
    // and never written out)
    const int c = tid % PIECES * 4, first = tid / PIECES;
    const float* src[NP];
#pragma unroll
    for (int i = 0; i < NP; ++i) {
        const int r = first + i * STEP;
        src[i] = (r < FB ? W + (size_t)min(n0 + r, p.N - 1) * p.ldw : A + (size_t)min(row0 + r - FB, p.M - 1) * p.lda) + c;
    }
    float* const dst = ring + first * LD + c;
    auto request = [&](int s, int stage) {
        if (s < slices) {
            const int k0 = s * KT;
            const bool inside = k0 + c < p.K;
#pragma unroll
            for (int i = 0; i < NP; ++i)
                if ((FB + ROWS) % STEP == 0 || first + i * STEP < FB + ROWS)
                    cp_async16(dst + stage * STAGE_FLOATS + i * STEP * LD, src[i] + (inside ? k0 : -c), inside);
        }
        cp_async_commit();
    };
    float acc[RB];
#pragma unroll
    for (int r = 0; r < RB; ++r) acc[r] = 0.f;
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) request(s, s);
    const int f = tid % FB, g = tid / FB;
    const bool computes = FB * ROWS / RB == THREADS || tid < FB * ROWS / RB;
    int stage = 0;
    for (int s = 0; s < slices; ++s) {
        cp_async_wait<STAGES - 2>();
        __syncthreads();
        request(s + STAGES - 1, stage == 0 ? STAGES - 1 : stage - 1);      // into the stage that every thread was done with before this barrier
        if (computes) {
            const float* w = ring + stage * STAGE_FLOATS + f * LD;
            const float* x = ring + stage * STAGE_FLOATS + (FB + g * RB) * LD;
#pragma unroll
            for (int k = 0; k < KT; k += 4) {
                const float4 wv = *reinterpret_cast<const float4*>(w + k);
#pragma unroll
                for (int r = 0; r < RB; ++r) {
                    const float4 xv = *reinterpret_cast<const float4*>(x + r * LD + k);
                    acc[r] = fmaf(xv.x, wv.x, acc[r]);
                    acc[r] = fmaf(xv.y, wv.y, acc[r]);
                    acc[r] = fmaf(xv.z, wv.z, acc[r]);
                    acc[r] = fmaf(xv.w, wv.w, acc[r]);
                }
            }
        }
        stage = stage == STAGES - 1 ? 0 : stage + 1;
    }
    if (computes && n0 + f < p.N) {
#pragma unroll
        for (int r = 0; r < RB; ++r) {
            const int m = row0 + g * RB + r;
            if (m < p.M) C[(size_t)m * p.ldc + n0 + f] = acc[r];
        }
    }
    pdl_trigger();
}

template <int FB, int ROWS, int RB, int KT, int STAGES>
int launch_few_rows(const Product& p, int batch, cudaStream_t stream) {
    constexpr int smem = STAGES * (FB + ROWS) * (KT + 4) * (int)sizeof(float);
    const cudaError_t e = cudaFuncSetAttribute(sgemm_few_rows_kernel<FB, ROWS, RB, KT, STAGES>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    rlis_launch(sgemm_few_rows_kernel<FB, ROWS, RB, KT, STAGES>, dim3((p.N + FB - 1) / FB, (p.M + ROWS - 1) / ROWS, batch),
                FewRows<FB, ROWS, RB>::THREADS, smem, stream, p);
    return RLIS_LAUNCH_CHECK();
}

template <int BM, int BN>
int launch_tiles(const Product& p, int batch, bool vec, cudaStream_t stream) {
    const dim3 grid((p.N + BN - 1) / BN, (p.M + BM - 1) / BM, batch);
    if (grid.y > 65535 || grid.z > 65535) return RLIS_ERR_UNSUPPORTED;
    if (vec)
        rlis_launch(sgemm_nt_kernel<BM, BN, true>, grid, TILE_THREADS, 0, stream, p);
    else
        rlis_launch(sgemm_nt_kernel<BM, BN, false>, grid, TILE_THREADS, 0, stream, p);
    return RLIS_LAUNCH_CHECK();
}

// A product in CTAs of few rows: 16 features a CTA while one such CTA an SM covers N, 32 while those leave each SM
// fewer than about three, else 64 and more, whose threads share what they read from shared memory among
// more outputs.  (8 rows, K 2048: N 2048 11.5 us with 16 features a CTA, 16.2 with 32; N 3072 19.2 and 16.4;
// N 16384 68 with 16, 69 with 32, 43 with 64.)
template <int ROWS> int run_few_rows(const Product& p, int batch, int sms, cudaStream_t stream) {
    const long long n = (long long)p.N * batch;
    constexpr int SMALL = ROWS <= 8 ? 256 : 128;        // k of a slice
    if (n <= 16LL * sms) return launch_few_rows<16, ROWS, (ROWS < 16 ? 1 : ROWS / 8), SMALL, (SMALL == 256 ? 4 : 6)>(p, batch, stream);
    if (n <= 64LL * sms) return launch_few_rows<32, ROWS, (ROWS < 8 ? 1 : ROWS == 32 ? 4 : 2), 64, 6>(p, batch, stream);
    if constexpr (ROWS == 1) return launch_few_rows<128, 1, 1, 64, 3>(p, batch, stream);
    else if constexpr (ROWS == 4) return launch_few_rows<128, 4, 4, 32, 4>(p, batch, stream);
    else if constexpr (ROWS == 8) return launch_few_rows<64, 8, 4, 64, 4>(p, batch, stream);
    else return launch_few_rows<64, ROWS, 8, 32, 6>(p, batch, stream);
}

// How long `ctas` CTAs take that need `alone` each on an SM of their own and `shared` of that when several share one.
inline double cta_time(long long ctas, int sms, double alone, double shared) {
    const long long per = (ctas + sms - 1) / sms;
    return per <= 1 ? alone : alone * shared * per;
}

// Which kernel a product goes to.  FEW: a step's few rows; else the split of the outputs that takes least time on this many SMs, by what a CTA of each
// kind was measured to take (us at K 2048 alone on an SM; all are proportional to K).  The more outputs a CTA has, the less it
// takes for each, and the fewer SMs a small product occupies.
enum Shape { FEW, ROWS_32x64, ROWS_32x32, TILE_128x128, TILE_128x64, TILE_64x64, SHAPES };

Shape choose(int M, int N, int batch, bool vec, int sms) {
    if (vec && M <= 32) return FEW;
    auto ctas = [&](int bm, int bn) { return (((long long)M + bm - 1) / bm) * (((long long)N + bn - 1) / bn) * batch; };
    const double t128 = cta_time(ctas(128, 128), sms, 211, 0.9), t128x64 = cta_time(ctas(128, 64), sms, 137, 0.83),
                 t64 = cta_time(ctas(64, 64), sms, 92, 0.97);
    if (vec && M <= 32 * 65535) {
        const double f64 = cta_time(ctas(32, 64), sms, 57, 1.0), f32 = cta_time(ctas(32, 32), sms, 35, 1.0);
        if (f64 < t128 && f64 < t128x64 && f64 < t64 && f64 <= f32) return ROWS_32x64;
        if (f32 < t128 && f32 < t128x64 && f32 < t64) return ROWS_32x32;
    }
    return t128 <= t128x64 && t128 <= t64 ? TILE_128x128 : t128x64 <= t64 ? TILE_128x64 : TILE_64x64;
}

int run(const Product& p, int batch, cudaStream_t stream) {
    if (p.M <= 0 || p.N <= 0 || batch <= 0) return 0;
    if (batch > 65535) return RLIS_ERR_UNSUPPORTED;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // 16-byte loads need rows and pieces of k on 16-byte boundaries
    const bool vec = p.K > 0 && p.K % 4 == 0 && p.lda % 4 == 0 && p.ldw % 4 == 0 && p.sa % 4 == 0 && p.sw % 4 == 0 &&
                     ((reinterpret_cast<uintptr_t>(p.A) | reinterpret_cast<uintptr_t>(p.W)) & 15) == 0;
    switch (choose(p.M, p.N, batch, vec, sms)) {
        case FEW:
            if (p.M == 1) return run_few_rows<1>(p, batch, sms, stream);
            if (p.M <= 4) return run_few_rows<4>(p, batch, sms, stream);
            if (p.M <= 8) return run_few_rows<8>(p, batch, sms, stream);
            if (p.M <= 16) return run_few_rows<16>(p, batch, sms, stream);
            return run_few_rows<32>(p, batch, sms, stream);
        case ROWS_32x64: return launch_few_rows<64, 32, 8, 32, 6>(p, batch, stream);
        case ROWS_32x32: return launch_few_rows<32, 32, 4, 64, 6>(p, batch, stream);
        case TILE_128x128: return launch_tiles<128, 128>(p, batch, vec, stream);
        case TILE_128x64: return launch_tiles<128, 64>(p, batch, vec, stream);
        default: return launch_tiles<64, 64>(p, batch, vec, stream);
    }
}
}  // namespace

extern "C" int rlis_gemm_f32_nt(const float* A, const float* W, float* C, int M, int N, int K,
                                cudaStream_t stream) {
    return run({A, W, C, M, N, K, K, K, N, 0, 0, 0}, 1, stream);
}

// `batch` products of the same sizes: entry b reads A + b * sa (rows lda apart), W + b * sw (rows ldw
// apart) and writes C + b * sc (rows ldc apart); strides in elements.  The per-head maps of a mixer.
extern "C" int rlis_gemm_f32_nt_batched(const float* A, const float* W, float* C, int M, int N, int K,
                                        long long lda, long long ldw, long long ldc, int batch, long long sa,
                                        long long sw, long long sc, cudaStream_t stream) {
    return run({A, W, C, M, N, K, lda, ldw, ldc, sa, sw, sc}, batch, stream);
}

// The kernel that a product of M x N outputs goes to on a device of `sms` SMs (`aligned`: rows and k on 16-byte boundaries), as a number below
// rlis_gemm_f32_shapes(): what tests cover the kernels by.
extern "C" int rlis_gemm_f32_shape(int M, int N, int batch, int aligned, int sms) {
    return M <= 0 || N <= 0 || batch <= 0 || sms <= 0 ? -1 : (int)choose(M, N, batch, aligned != 0, sms);
}
extern "C" int rlis_gemm_f32_shapes(void) { return (int)SHAPES; }
