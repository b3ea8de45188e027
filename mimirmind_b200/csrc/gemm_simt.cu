// C[M,N] = A[M,K] * W[N,K]^T (+ bias[N]) on the fp32 FMA units: the any-shape product of the true 32-bit path
// (its layers' weights go to gemm_split_tcgen05.cu) and the fallback of the bfloat16 path.
//
// The reference computes Y[m,n] = sum_k X[m,k] * W[n,k] with W stored [N_out, K_in]
// (src/compute/Matmul.cpp:54-65) and adds a bias per output column
// (src/compute/Matmul.cpp:67-78).  Every output element is accumulated over k in
// ascending order by one thread, so its value does not depend on M, on the row's place
// in the batch, on the tile it falls into, or on which of the two kernels below made it.
#include "common.cuh"
#include "gemm_split.h"

// ---------------------------------------------------------------------------------------------------------------
// tiles: a thread owns TM x TN outputs
// ---------------------------------------------------------------------------------------------------------------
// Bound by the FMA units and what feeds them.  Two rows' products are one packed instruction (each half rounds as the plain
// one does), the numbers of the next k are read from shared memory while the current ones are multiplied, and the next BK
// of both operands are on their way from global memory into registers meanwhile (two buffers, one barrier per BK).
// A buffer is [k][row]; a row's place is turned by (k / 4 % 8) * 4, so that the scattered stores of a warp (8 runs of k x 4
// rows) fall into 32 different banks and four neighbouring rows still are one 16-byte word.
// 64 x 64 outputs of 128 threads (8 x 4 each): 40.9 TFLOP/s where they fill the GPU (509 x 9,728 x 896 in 217 us, 4 x 4 a thread with
// scalar loads 477).  Larger tiles (128 x 64, 128 x 128 of
// 8 x 8) gain nothing where they fill the GPU and lose a factor of 2 and 3 where they do not; fp32 FMAs alone: 10 % slower.
template <typename T, bool VEC>
__device__ __forceinline__ float4 simt_load4(const T* __restrict__ p, bool row_ok, int k, int K) {     // VEC: one aligned load, K % 4 == 0
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (!row_ok) return v;
    if (VEC) {
        if (k < K) {
            if (sizeof(T) == 4) {
                v = *reinterpret_cast<const float4*>(p + k);
            } else {
                const uint2 u = *reinterpret_cast<const uint2*>(p + k);
                v = make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16),
                                __uint_as_float(u.y & 0xffff0000u));
            }
        }
    } else {
        if (k < K) v.x = to_f32<T>(p[k]);
        if (k + 1 < K) v.y = to_f32<T>(p[k + 1]);
        if (k + 2 < K) v.z = to_f32<T>(p[k + 2]);
        if (k + 3 < K) v.w = to_f32<T>(p[k + 3]);
    }
    return v;
}

template <typename TA, typename TW, typename TC, int BM, int BN, int TM, int TN, int BK, bool VEC>
__global__ void __launch_bounds__((BM / TM) * (BN / TN)) gemm_simt_kernel(const TA* __restrict__ A, const TW* __restrict__ W,
                                                                          const void* __restrict__ bias, int bias_dtype,
                                                                          TC* __restrict__ C, int M, int N, int K, int lda, int ldc) {
    constexpr int THREADS = (BM / TM) * (BN / TN), TX = BN / TN, KQ = BK / 4;
    constexpr int LA = BM * KQ / THREADS, LW = BN * KQ / THREADS;      // runs of four k that a thread fetches
    constexpr int STAGE = BK * (BM + BN);
    static_assert(BM * KQ % THREADS == 0 && BN * KQ % THREADS == 0 && TM % 4 == 0 && TN % 4 == 0 && BM >= 32 && BN >= 32, "tile");
    extern __shared__ __align__(16) float simt_smem[];
    const int tid = threadIdx.x;
    const int tx = tid % TX, ty = tid / TX;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    uint64_t acc[TM / 2][TN];                    // two rows each
#pragma unroll
    for (int i = 0; i < TM / 2; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;

    float4 ra[LA], rw[LW];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int e = 0; e < LA; ++e) {
            const int idx = tid + e * THREADS, r = idx / KQ, k = k0 + (idx % KQ) * 4;
            ra[e] = simt_load4<TA, VEC>(A + (size_t)(m0 + r) * lda, m0 + r < M, k, K);
        }
#pragma unroll
        for (int e = 0; e < LW; ++e) {
            const int idx = tid + e * THREADS, r = idx / KQ, k = k0 + (idx % KQ) * 4;
            rw[e] = simt_load4<TW, VEC>(W + (size_t)(n0 + r) * K, n0 + r < N, k, K);
        }
    };
    auto place = [&](int buf) {
        float* sa = simt_smem + buf * STAGE;
        float* sw = sa + BK * BM;
#pragma unroll
        for (int e = 0; e < LA; ++e) {
            const int idx = tid + e * THREADS, r = idx / KQ, q = idx % KQ, at = q * 4 * BM + (r ^ ((q & 7) << 2));
            sa[at] = ra[e].x;
            sa[at + BM] = ra[e].y;
            sa[at + 2 * BM] = ra[e].z;
            sa[at + 3 * BM] = ra[e].w;
        }
#pragma unroll
        for (int e = 0; e < LW; ++e) {
            const int idx = tid + e * THREADS, r = idx / KQ, q = idx % KQ, at = q * 4 * BN + (r ^ ((q & 7) << 2));
            sw[at] = rw[e].x;
            sw[at + BN] = rw[e].y;
            sw[at + 2 * BN] = rw[e].z;
            sw[at + 3 * BN] = rw[e].w;
        }
    };
    // a thread's columns: runs of four, TX * 4 apart, so that neighbouring threads read neighbouring 16-byte words
    auto column = [&](int j) { return (j >> 2) * (TX * 4) + tx * 4 + (j & 3); };
    auto read = [&](int buf, int kk, float* a, float* w) {
        const float* sa = simt_smem + buf * STAGE + kk * BM;
        const float* sw = simt_smem + buf * STAGE + BK * BM + kk * BN;
        const int turn = ((kk >> 2) & 7) << 2;
#pragma unroll
        for (int i = 0; i < TM; i += 4) {
            const float4 v = *reinterpret_cast<const float4*>(sa + ((ty * TM + i) ^ turn));
            a[i] = v.x; a[i + 1] = v.y; a[i + 2] = v.z; a[i + 3] = v.w;
        }
#pragma unroll
        for (int j = 0; j < TN; j += 4) {
            const float4 v = *reinterpret_cast<const float4*>(sw + (column(j) ^ turn));
            w[j] = v.x; w[j + 1] = v.y; w[j + 2] = v.z; w[j + 3] = v.w;
        }
    };

    fetch(0);
    place(0);
    __syncthreads();
    int buf = 0;
    for (int k0 = 0; k0 < K; k0 += BK, buf ^= 1) {
        const bool more = k0 + BK < K;
        if (more) fetch(k0 + BK);
        float a[2][TM], w[2][TN];
        read(buf, 0, a[0], w[0]);
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            if (kk + 1 < BK) read(buf, kk + 1, a[(kk + 1) & 1], w[(kk + 1) & 1]);
            uint64_t pa[TM / 2];
#pragma unroll
            for (int i = 0; i < TM / 2; ++i)
                asm("mov.b64 %0, {%1, %2};" : "=l"(pa[i]) : "r"(__float_as_uint(a[kk & 1][2 * i])), "r"(__float_as_uint(a[kk & 1][2 * i + 1])));
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                uint64_t pw;
                asm("mov.b64 %0, {%1, %1};" : "=l"(pw) : "r"(__float_as_uint(w[kk & 1][j])));
#pragma unroll
                for (int i = 0; i < TM / 2; ++i) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i][j]) : "l"(pa[i]), "l"(pw));
            }
        }
        if (more) {
            place(buf ^ 1);          // the buffer read before the barrier that ended the step before
            __syncthreads();
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + ty * TM + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + column(j);
            if (n >= N) continue;
            float v = __uint_as_float((uint32_t)(acc[i / 2][j] >> (32 * (i & 1))));
            if (bias) {
                v += (bias_dtype == MM_F32) ? ((const float*)bias)[n] : __bfloat162float(((const __nv_bfloat16*)bias)[n]);
            }
            C[(size_t)m * ldc + n] = from_f32<TC>(v);
        }
    }
}

// ---------------------------------------------------------------------------------------------------------------
// a few rows of fp32: the weights are streamed once
// ---------------------------------------------------------------------------------------------------------------
// Bound by reading W.  A block owns NB rows of W and walks k in chunks of KB numbers that asynchronous copies bring into a ring of
// STAGES buffers; thread (c, g) of the 128 owns column c and the rows g, g + 128/NB, ... of A, R of them, and adds up k in
// order.  A row of a buffer is padded by 16 bytes: the eight threads of a quarter warp read eight different bank groups.
// 4 rows: 151,936 x 896 (545 MB) in 104 us with 128 rows of W per block, where a number of W is read once from shared memory (142 us with 32,
// where each of 4 row groups reads it; 64-row tiles, the form before: 879).
#define SIMT_GEMV_ROWS 16

__device__ __forceinline__ void simt_cp16(void* smem, const void* gmem, bool in) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(smem);
    const int bytes = in ? 16 : 0;               // 0: the 16 bytes are filled with zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(gmem), "r"(bytes));
}

template <int NB, int KB, int STAGES, int R>
__global__ void __launch_bounds__(128) gemv_simt_kernel(const float* __restrict__ A, const float* __restrict__ W,
                                                        const void* __restrict__ bias, int bias_dtype, float* __restrict__ C, int M, int N,
                                                        int K, int lda, int ldc) {
    constexpr int G = 128 / NB, LD = KB + 4, KQ = KB / 4, UNROLL = KQ < 16 ? KQ : 16;
    extern __shared__ __align__(16) float simt_smem[];
    const int stage = (NB + M) * LD;             // floats of one buffer: NB rows of W, then the M rows of A
    const int tid = threadIdx.x, c = tid % NB, g = tid / NB;
    const int n0 = blockIdx.x * NB;
    auto fill = [&](int chunk) {
        float* s = simt_smem + (chunk % STAGES) * stage;
        const int k0 = chunk * KB;
#pragma unroll
        for (int e = 0; e < NB * KQ / 128; ++e) {
            const int idx = tid + e * 128, r = idx / KQ, kq = (idx % KQ) * 4;
            const int n = min(n0 + r, N - 1);
            const bool in = k0 + kq < K;
            simt_cp16(s + r * LD + kq, W + (size_t)n * K + (in ? k0 + kq : 0), in);
        }
        for (int idx = tid; idx < M * KQ; idx += 128) {
            const int r = idx / KQ, kq = (idx % KQ) * 4;
            const bool in = k0 + kq < K;
            simt_cp16(s + (NB + r) * LD + kq, A + (size_t)r * lda + (in ? k0 + kq : 0), in);
        }
    };
    const int chunks = (K + KB - 1) / KB;
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < chunks) fill(s);
        asm volatile("cp.async.commit_group;\n" ::);
    }
    float acc[R];
#pragma unroll
    for (int i = 0; i < R; ++i) acc[i] = 0.0f;
    for (int ch = 0; ch < chunks; ++ch) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2));
        __syncthreads();                         // chunk ch has landed for every thread, and nobody still reads chunk ch - 1
        if (ch + STAGES - 1 < chunks) fill(ch + STAGES - 1);
        asm volatile("cp.async.commit_group;\n" ::);
        const float* sw = simt_smem + (ch % STAGES) * stage + c * LD;
        const float* sa = simt_smem + (ch % STAGES) * stage + NB * LD;
        auto step = [&](int k) {
            const float4 w = *reinterpret_cast<const float4*>(sw + k);
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const int m = min(g + i * G, M - 1);
                const float4 a = *reinterpret_cast<const float4*>(sa + m * LD + k);
                acc[i] = fmaf(a.x, w.x, acc[i]);
                acc[i] = fmaf(a.y, w.y, acc[i]);
                acc[i] = fmaf(a.z, w.z, acc[i]);
                acc[i] = fmaf(a.w, w.w, acc[i]);
            }
        };
        if (g < M) {
            const int len = K - ch * KB;         // a multiple of 4
            if (len >= KB) {
#pragma unroll UNROLL
                for (int k = 0; k < KB; k += 4) step(k);
            } else {
                for (int k = 0; k < len; k += 4) step(k);
            }
        }
    }
    const int n = n0 + c;
    if (n >= N) return;
    float b = 0.0f;
    if (bias) b = (bias_dtype == MM_F32) ? ((const float*)bias)[n] : __bfloat162float(((const __nv_bfloat16*)bias)[n]);
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int m = g + i * G;
        if (m < M) C[(size_t)m * ldc + n] = bias ? acc[i] + b : acc[i];
    }
}

template <int NB, int KB, int STAGES, int R>
static int launch_gemv_simt(const void* A, const void* W, const void* bias, int bias_dtype, void* C, int M, int N, int K, int lda, int ldc,
                            cudaStream_t s) {
    const size_t smem = (size_t)STAGES * (NB + M) * (KB + 4) * sizeof(float);
    constexpr size_t most = (size_t)STAGES * (NB + SIMT_GEMV_ROWS) * (KB + 4) * sizeof(float);
    if (!mm_allow_smem<gemv_simt_kernel<NB, KB, STAGES, R>>(most)) {
        mm_set_last_error("gemm: cannot reserve shared memory");
        return MM_ERR_LAUNCH;
    }
    mm_launch(gemv_simt_kernel<NB, KB, STAGES, R>, dim3(ceil_div(N, NB)), dim3(128), smem, s, (const float*)A, (const float*)W, bias, bias_dtype,
              (float*)C, M, N, K, lda, ldc);
    MM_CHECK_LAUNCH();
    return MM_OK;
}

template <typename TA, typename TW, typename TC, int BM, int BN, int TM, int TN, int BK, bool VEC>
static int launch_simt_tile(const void* A, const void* W, const void* bias, int bias_dtype, void* C, int M, int N, int K, int lda, int ldc,
                            cudaStream_t s) {
    const int smem = 2 * BK * (BM + BN) * (int)sizeof(float);
    if (smem > 48 * 1024 && !mm_allow_smem<gemm_simt_kernel<TA, TW, TC, BM, BN, TM, TN, BK, VEC>>(smem)) {
        mm_set_last_error("gemm: cannot reserve shared memory");
        return MM_ERR_LAUNCH;
    }
    mm_launch(gemm_simt_kernel<TA, TW, TC, BM, BN, TM, TN, BK, VEC>, dim3(ceil_div(N, BN), ceil_div(M, BM)), dim3((BM / TM) * (BN / TN)), (size_t)smem,
              s, (const TA*)A, (const TW*)W, bias, bias_dtype, (TC*)C, M, N, K, lda, ldc);
    MM_CHECK_LAUNCH();
    return MM_OK;
}

template <typename TA, typename TW, typename TC>
static int launch_gemm_simt(const void* A, const void* W, const void* bias, int bias_dtype, void* C, int M, int N, int K, int lda, int ldc,
                            cudaStream_t s) {
    const bool vec = K % 4 == 0 && lda % 4 == 0 && (uintptr_t)A % (4 * sizeof(TA)) == 0 && (uintptr_t)W % (4 * sizeof(TW)) == 0;
#define SIMT_TILE(BM, TM, BK)                                                                                                            \
    return vec ? launch_simt_tile<TA, TW, TC, BM, 64, TM, 4, BK, true>(A, W, bias, bias_dtype, C, M, N, K, lda, ldc, s)                    \
               : launch_simt_tile<TA, TW, TC, BM, 64, TM, 4, BK, false>(A, W, bias, bias_dtype, C, M, N, K, lda, ldc, s)
    // 32-row tiles where they put fewer rows on the busiest SM (or M does not fill 64): 100 x 1,152 x 512 15.1 us against 17.0; where both
    // put the same, 64 rows are ahead (1,000 x 512 x 512 17.7 against 21.4, 5,000 x 64 x 2,048 61.7 against 80.9).  With at most two blocks per SM there is
    // no other block to fill the barriers, and the deeper step pays (17.7 against 30.8, 61.7 against 116.7; with more blocks 4,000 x 1,024 x 512 97.5 and 96.9).
    const long long rounds64 = ceil_div(ceil_div(M, 64) * (long long)ceil_div(N, 64), 148);
    const long long rounds32 = ceil_div(ceil_div(M, 32) * (long long)ceil_div(N, 64), 148);
    if (M <= 32 * 65535 && (M <= 32 || rounds32 * 32 * 10 <= rounds64 * 64 * 8)) SIMT_TILE(32, 4, 32);
    if constexpr (sizeof(TA) == 4 && sizeof(TW) == 4 && sizeof(TC) == 4)
        if (vec && rounds64 <= 2) return launch_simt_tile<TA, TW, TC, 64, 64, 8, 4, 64, true>(A, W, bias, bias_dtype, C, M, N, K, lda, ldc, s);
    SIMT_TILE(64, 8, 32);
#undef SIMT_TILE
}

// err: device int set to 1 when a bounded wait of the tensor-core form ran out (may be null)
MM_EXPORT int mm_gemm_simt(const void* A, int a_dtype, const void* W, int w_dtype, const void* bias, int bias_dtype,
                           void* C, int c_dtype, int M, int N, int K, int lda, int ldc, void* err, void* stream) {
    MM_REQUIRE(M >= 0 && N > 0 && K > 0 && lda >= K && ldc >= N, "gemm: bad sizes");
    if (M == 0) return MM_OK;
    cudaStream_t s = (cudaStream_t)stream;
    typedef __nv_bfloat16 bf;
    const int key = a_dtype * 4 + w_dtype * 2 + c_dtype;
    if (key == 0 && gemm_split_takes(W, N, K)) return gemm_split((const float*)A, (const float*)W, bias, bias_dtype, (float*)C, M, N, K, lda, ldc, (int*)err, s);
    if (key == 0 && M <= SIMT_GEMV_ROWS && K % 4 == 0 && lda % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0) {
#define SIMT_GEMV(NB, KB, STAGES, R) return launch_gemv_simt<NB, KB, STAGES, R>(A, W, bias, bias_dtype, C, M, N, K, lda, ldc, s)
        // as many rows of W per block as still leave every SM a few blocks
        if (N >= 2 * 148 * 128) {
            if (M <= 1) SIMT_GEMV(128, 32, 4, 1);
            if (M <= 2) SIMT_GEMV(128, 32, 4, 2);
            if (M <= 4) SIMT_GEMV(128, 32, 4, 4);
            if (M <= 8) SIMT_GEMV(128, 32, 4, 8);
            SIMT_GEMV(128, 32, 4, 16);
        }
        if (N >= 2 * 148 * 16) {
            if (M <= 8) SIMT_GEMV(16, 128, 4, 1);
            SIMT_GEMV(16, 128, 4, 2);
        }
        SIMT_GEMV(8, 256, 6, 1);
#undef SIMT_GEMV
    }
#define MM_GEMM(TA, TW, TC) return launch_gemm_simt<TA, TW, TC>(A, W, bias, bias_dtype, C, M, N, K, lda, ldc, s)
    switch (key) {
        case 0: MM_GEMM(float, float, float);
        case 1: MM_GEMM(float, float, bf);
        case 2: MM_GEMM(float, bf, float);
        case 3: MM_GEMM(float, bf, bf);
        case 4: MM_GEMM(bf, float, float);
        case 5: MM_GEMM(bf, float, bf);
        case 6: MM_GEMM(bf, bf, float);
        case 7: MM_GEMM(bf, bf, bf);
        default: break;
    }
#undef MM_GEMM
    MM_REQUIRE(false, "gemm: dtypes must be float32 or bfloat16");
}
