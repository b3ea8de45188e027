// C[M,N] = A[M,K] * W[N,K]^T (+ bias[N]) in float32 on the fifth-generation tensor cores: the product of the true 32-bit path for
// the weights of layers (see gemm_split_takes).
//
// Every number is split into three bf16 numbers, which hold all of its 24 bits, and a product is the sum of the six larger of the nine partial
// products (Henry, Tang and Heinecke 2019).  bf16 ends at 2^-133, so the numbers are multiplied by 2^16 before (the third part of a
// number below 2^-110 would be cut off otherwise) and the results by 2^-32 in the end, which changes no bit of what both ways hold.  The
// tensor core cuts off what falls below 2^-24 of a sum's largest term instead of rounding, so the largest partial products, which have 16 bits, are summed there sixteen k at a time from zero and added up beyond that by rounded additions;
// the five others, 2^-8 of them, stay on the tensor core for a part of k.  Error against 64 bits in 1e-7 of the result's size (2-norm):
// 0.87 for K = 896, 1.30 for 4,864 and 2.4 for 18,944, where FMAs over k in ascending order have 5.3, 12.5 and 25.
//
// Which sums are made, and in which order, follows from K alone: k is cut into up to eight parts (gemm_split_parts), a part's sums are added up
// in order, the parts' results in order.  The tile's size along the tokens and whether the parts are walked by one CTA or shared out over a
// cluster do not change a bit, so a row's value depends neither on M nor on what stands beside it.  (For up to 16 tokens that rests on mma.sync
// and tcgen05.mma adding sixteen products up to the same bits.  They do, as far as the tests look, with operands up to 2^60 apart; no document
// says that they have to.)  A result that is not finite (an
// operand was not, or is 2^112 or more, or a sum reached 2^96) is made again by FMAs over k in ascending order (gs_again).
// All waits are bounded; when one runs out the CTA gives its tensor memory back, sets `err` and makes its whole tile again like that.
//
// A CTA works on 128 rows of W (M of the instruction) x NT tokens (its N), 64 k a step:
//   warps 0..7    bring both operands' 64 k in as fp32 (asynchronous copies that a thread later reads back itself, or registers), split them and
//                 write the three planes of each in the 128-byte swizzle;
//   warp 16       one thread issues tcgen05.mma: per sixteen k the largest products into one of HB buffers, the five others onto `low`;
//   warps 8..15   read each buffer back and add it up (32 rows and half of the tokens a warp).
// Bound by nothing that is full: 1,024 x 9,728 x 896, 608 tiles of 128 tokens on 148 SMs, keeps an SM at work for 79 % of the time (the fifth round holds 16
// tiles), and then its issue slots are busy for 63 % (splitting and summing), shared memory for 48 % (a step reads 192 KB of it for the tensor core
// and writes 96 KB of planes), the tensor cores for less; the rest goes into what the roles hand over.  From graphs of 20 launches, us: 509 x 9,728 x 896 95.8 (93 TFLOP/s of
// 32-bit products; by FMAs 217), 1,024 x 9,728 x 896 159 (397), 509 x 896 x 4,864, eight CTAs to a tile, 51.7 (142).  The issuing warp walks along converged and elects its thread: with one lane in a branch of
// its own a product took 170 clocks to issue instead of the 39 (16 tokens) to 64 (128) that it runs.
#include "tcgen05.cuh"
#include "gemm_split.h"

namespace {

using namespace tc;

constexpr int SPLIT_WARPS = 8, SUM_WARPS = 8, SPLIT_THREADS = 32 * (SPLIT_WARPS + SUM_WARPS + 1);
constexpr int W_PLANE = 128 * 128;            // bytes: 128 rows of 64 bf16

template <int NT>
struct SplitShape {
    static constexpr int X_PLANE = NT * 128;
    static constexpr int STAGE = 3 * (W_PLANE + X_PLANE);                   // both operands' planes of 64 k
    static constexpr int RING = NT == 32 ? 2 : 1;                                      // steps of fp32 on their way in shared memory
    static constexpr int RING_PIECES = NT == 128 ? 8 : (128 + NT) / 16;     // of a thread and step; what does not fit there waits in registers
    static constexpr int RING_BYTES = RING_PIECES * 4096;
    static constexpr int SMEM = 1024 + 2 * STAGE + RING * RING_BYTES;
    static constexpr int HB = NT == 128 ? 2 : 4;                            // buffers of the largest products: sixteen k each, handed over together
    static constexpr int COLS = NT >= 64 ? 512 : 8 * NT;                    // tensor memory: HB buffers, low, the parts' sum
    static constexpr int PIECES = (128 + NT) / 16;                          // runs of four k that a thread brings in per step
    static_assert((HB + 2) * NT <= COLS && NT * 512 <= 2 * STAGE, "tile");
};

struct SplitArgs {
    const float *A, *W;
    const void* bias;
    float* C;
    int bias_dtype, M, N, K, lda, ldc, parts, ranks;
    bool a_words;            // rows of A stand on 16-byte boundaries
    int* err;
    int give_up;             // 1: as if a wait had run out from the start, so that none is tried more than once
};

__device__ __forceinline__ uint32_t gs_round2(float x, float y) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(y), "f"(x));
    return r;
}
__device__ __forceinline__ void gs_rest(float& x, float& y, uint32_t part) {
    x = __fsub_rn(x, __uint_as_float(part << 16));
    y = __fsub_rn(y, __uint_as_float(part & 0xffff0000u));
}
__device__ __forceinline__ void gs_store8(uint32_t at, uint32_t x, uint32_t y) { asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at), "r"(x), "r"(y) : "memory"); }
// What is split is 2^16 times the number: see the header.
constexpr float GS_UP = 65536.0f, GS_DOWN = 1.0f / (65536.0f * 65536.0f);
__device__ __forceinline__ void gs_up2(float& x, float& y) {
    uint64_t v;
    asm("{\n\t.reg .b64 u;\n\tmov.b64 %0, {%1, %2};\n\tmov.b64 u, {%3, %3};\n\tmul.rn.f32x2 %0, %0, u;\n\t}" : "=&l"(v) : "f"(x), "f"(y), "f"(GS_UP));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
}
// four consecutive k of a row as the three planes
__device__ __forceinline__ void gs_split4(uint32_t at, int plane, float4 v) {
    gs_up2(v.x, v.y);
    gs_up2(v.z, v.w);
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        const uint32_t a = gs_round2(v.x, v.y), b = gs_round2(v.z, v.w);
        gs_store8(at + p * plane, a, b);
        gs_rest(v.x, v.y, a);
        gs_rest(v.z, v.w, b);
    }
}
template <int BYTES>
__device__ __forceinline__ void gs_copy(uint32_t to, const void* from, bool in) {
    const int bytes = in ? BYTES : 0;            // 0: filled with zeros
    if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(to), "l"(from), "r"(bytes) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(to), "l"(from), "r"(bytes) : "memory");
}

// CH columns of this warp's 32 lanes of tensor memory
template <int CH>
__device__ __forceinline__ void gs_ld(uint32_t at, float* v) {
    uint32_t r[CH];
    if constexpr (CH == 8) {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(at));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    } else if constexpr (CH == 16) {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                       "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(at));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    } else {
        tmem_ld32(at, r);
    }
#pragma unroll
    for (int i = 0; i < CH; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void gs_st8(uint32_t at, const float* v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(at), "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])),
                 "r"(__float_as_uint(v[2])), "r"(__float_as_uint(v[3])), "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])),
                 "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7])) : "memory");
}
// A bounded wait that sleeps in the barrier (up to 20 us a try, so under 2 s in all): seventeen warps that poll instead keep the
// stores of the planes waiting.  False when it ran out, here or in another warp; the lanes of a warp may see the one or the other, and what
// follows is for whole warps, so no lane leaves its way for it: the summing warps stop after a vote, the others walk on to their ends
// without waiting for more than a try.  The tile is made again then.
__device__ __forceinline__ bool gs_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    for (int it = 0; it < 100000; ++it) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(bar), "r"(parity), "r"(20000) : "memory");
        if (ok) return true;
        if (*abort_flag) return false;
    }
    *abort_flag = 1;
    return false;
}
__device__ __forceinline__ bool gs_elect() {
    uint32_t e;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(e));
    return e != 0;
}
__device__ __forceinline__ void gs_umma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ float4 gs_ld_cluster(uint32_t at) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at) : "memory");
    return v;
}
__device__ __forceinline__ void gs_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
// A result that the tensor cores have not given as a number: what 32-bit FMAs over k in order make of it, or, where that is a number (of 2^96 or
// more), 64-bit ones.  gs_again: a token's with ROWS rows of W (`rows` of them there), sixteen k of all rows on their way together, and no further
// once none of them is a number, which nothing changes.  A thread does it for itself, so it takes long where it takes many: 509 x 9,728 x 896
// with a NaN early in every row 211 us (what a state that has gone wrong brings, in every product from there on; one number and one k at a time it was
// 26,100), with an infinity in every row 10,000, with all results from 2^96 on 20,100.
__device__ __forceinline__ float gs_again64(const float* __restrict__ a, const float* __restrict__ w, int K) {
    double s = 0.0;
#pragma unroll 2
    for (int k = 0; k < K; k += 4) {
        const float4 y = __ldg(reinterpret_cast<const float4*>(w + k));
        s = fma((double)a[k], (double)y.x, s);
        s = fma((double)a[k + 1], (double)y.y, s);
        s = fma((double)a[k + 2], (double)y.z, s);
        s = fma((double)a[k + 3], (double)y.w, s);
    }
    return (float)s;
}
template <int ROWS>
__device__ __noinline__ float4 gs_again(const float* __restrict__ a, const float* __restrict__ w, int K, int rows, bool a_words) {
    const float* p[ROWS];
    float s[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        p[r] = w + (r < rows ? (size_t)r * K : 0);
        s[r] = 0.0f;
    }
    for (int k0 = 0; k0 < K; k0 += 16) {
        float4 x[4], y[ROWS][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k = k0 + 4 * i < K ? k0 + 4 * i : k0;
            x[i] = a_words ? __ldg(reinterpret_cast<const float4*>(a + k)) : make_float4(a[k], a[k + 1], a[k + 2], a[k + 3]);
#pragma unroll
            for (int r = 0; r < ROWS; ++r) y[r][i] = __ldg(reinterpret_cast<const float4*>(p[r] + k));
        }
        bool number = false;
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (k0 + 4 * i < K) {
                    s[r] = fmaf(x[i].x, y[r][i].x, s[r]);
                    s[r] = fmaf(x[i].y, y[r][i].y, s[r]);
                    s[r] = fmaf(x[i].z, y[r][i].z, s[r]);
                    s[r] = fmaf(x[i].w, y[r][i].w, s[r]);
                }
            number |= s[r] == s[r];
        }
        if (!number) break;
    }
#pragma unroll
    for (int r = 0; r < ROWS; ++r)
        if (isfinite(s[r])) s[r] = gs_again64(a, p[r], K);
    return make_float4(s[0], s[ROWS > 1 ? 1 : 0], s[ROWS > 2 ? 2 : 0], s[ROWS > 3 ? 3 : 0]);
}

struct SplitCtl {
    uint64_t full[2], empty[2];       // planes
    uint64_t sum_full, sum_empty;     // the HB buffers
    uint64_t low_full, low_empty;
    uint32_t tmem_base;
    int abort_flag;
};

template <int NT>
__global__ void __launch_bounds__(SPLIT_THREADS, 1) gemm_split_kernel(const SplitArgs g) {
    using S = SplitShape<NT>;
    constexpr int HB = S::HB;
    extern __shared__ unsigned char smem_raw[];
    __shared__ SplitCtl ctl;
    const uint32_t planes = (smem_u32(smem_raw) + 1023u) & ~1023u;          // the swizzle's unit is 1,024 bytes
    const uint32_t ring = planes + 2 * S::STAGE;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = blockIdx.x % g.ranks, m0 = (blockIdx.x / g.ranks) * NT, n0 = blockIdx.y * 128;
    const int steps = (g.K + 63) / 64;
    auto part_begin = [&](int p) { return (int)((long long)p * steps / g.parts); };
    // this CTA's parts: all of them, or part `rank`
    const int p_begin = g.ranks == 1 ? 0 : rank, p_end = g.ranks == 1 ? g.parts : rank + 1;
    const int first = part_begin(p_begin), last = part_begin(p_end);
    volatile int* abort_flag = &ctl.abort_flag;

    if (tid == 0) {
        for (int s = 0; s < 2; ++s) {
            mbar_init(smem_u32(&ctl.full[s]), SPLIT_WARPS);
            mbar_init(smem_u32(&ctl.empty[s]), 1);
        }
        mbar_init(smem_u32(&ctl.sum_full), 1);
        mbar_init(smem_u32(&ctl.sum_empty), SUM_WARPS);
        mbar_init(smem_u32(&ctl.low_full), 1);
        mbar_init(smem_u32(&ctl.low_empty), SUM_WARPS);
        ctl.abort_flag = g.give_up;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 16) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl.tmem_base)), "r"(S::COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = ctl.tmem_base;

    if (warp < SPLIT_WARPS) {
        // ---- operands: thread (row r0 + 16 e, four k at 4 q) of W's 128 rows and then of A's NT ----
        const int r0 = tid >> 4, q = tid & 15;
        const uint32_t place = r0 * 128 + ((((q >> 1) ^ (r0 & 7))) << 4) + (q & 1) * 8;
        const int w_rows = g.N - n0 - r0, a_rows = g.M - m0 - r0;
        const size_t w_next = 16 * (size_t)g.K, a_next = 16 * (size_t)g.lda;
        constexpr int HELD = S::PIECES - S::RING_PIECES;
        float4 v[HELD > 0 ? HELD : 1];
        auto fetch = [&](int step) {
            const int k = step * 64 + q * 4;
            const bool k_ok = k < g.K && step < last;
            const float *pw = g.W + (size_t)(n0 + r0) * g.K + k, *pa = g.A + (size_t)(m0 + r0) * g.lda + k;
#pragma unroll
            for (int e = 0; e < S::PIECES; ++e) {
                const bool is_w = e < 8;
                const bool in = k_ok && (is_w ? e * 16 < w_rows : (e - 8) * 16 < a_rows);
                const float* p = in ? (is_w ? pw : pa) : g.W;
                if (is_w) pw += w_next;
                else pa += a_next;
                if (e < S::RING_PIECES) {
                    const uint32_t to = ring + (step - first) % S::RING * S::RING_BYTES + (tid + e * 256) * 16;
                    if (is_w || g.a_words) {
                        gs_copy<16>(to, p, in);
                    } else {
#pragma unroll
                        for (int x = 0; x < 4; ++x) gs_copy<4>(to + 4 * x, in ? p + x : p, in);
                    }
                } else {
                    float4& x = v[e - S::RING_PIECES];
                    x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    if (in) x = g.a_words ? __ldg(reinterpret_cast<const float4*>(p)) : make_float4(p[0], p[1], p[2], p[3]);
                }
            }
            asm volatile("cp.async.commit_group;\n" ::: "memory");
        };
#pragma unroll
        for (int i = 0; i < S::RING; ++i) fetch(first + i);
        for (int step = first; step < last; ++step) {
            const int it = step - first, s = it & 1;
            gs_wait(smem_u32(&ctl.empty[s]), ((it >> 1) & 1) ^ 1, abort_flag);
            asm volatile("cp.async.wait_group %0;\n" ::"n"(S::RING - 1) : "memory");
            const uint32_t to = planes + s * S::STAGE + place;
            const float4* held = reinterpret_cast<const float4*>(smem_raw + (ring - smem_u32(smem_raw)) + it % S::RING * S::RING_BYTES) + tid;
            constexpr int BATCH = 4;
#pragma unroll
            for (int e0 = 0; e0 < S::PIECES; e0 += BATCH) {
                float4 x[BATCH];
#pragma unroll
                for (int e = e0; e < e0 + BATCH; ++e)
                    if (e < S::PIECES) x[e - e0] = e < S::RING_PIECES ? held[e * 256] : v[e < S::RING_PIECES ? 0 : e - S::RING_PIECES];
#pragma unroll
                for (int e = e0; e < e0 + BATCH; ++e) {
                    if (e < 8) gs_split4(to + e * 2048, W_PLANE, x[e - e0]);
                    else if (e < S::PIECES) gs_split4(to + 3 * W_PLANE + (e - 8) * 2048, S::X_PLANE, x[e - e0]);
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&ctl.full[s]));
            fetch(step + S::RING);
        }
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    } else if (warp < SPLIT_WARPS + SUM_WARPS) {
        // ---- sums: lanes 32 (warp % 4).., half of the tokens ----
        constexpr int CH = NT / 2, LD = NT == 128 ? 16 : CH;
        const int quarter = warp & 3, half = (warp - SPLIT_WARPS) >> 2;
        const uint32_t mine = tmem + ((uint32_t)(quarter * 32) << 16) + half * CH;
        float acc[CH];
        bool ok = true;
        int group = 0;
        for (int p = p_begin; p < p_end && ok; ++p) {
#pragma unroll
            for (int i = 0; i < CH; ++i) acc[i] = 0.0f;
            const int count = 4 / HB * (part_begin(p + 1) - part_begin(p));
#pragma unroll 1
            for (int c = 0; c < count; ++c, ++group) {
                if (!__all_sync(0xffffffffu, gs_wait(smem_u32(&ctl.sum_full), group & 1, abort_flag))) { ok = false; break; }
                tc_fence_after();
#pragma unroll
                for (int b = 0; b < HB; ++b)
#pragma unroll
                    for (int j = 0; j < CH; j += LD) {
                        float t[LD];
                        gs_ld<LD>(mine + b * NT + j, t);
#pragma unroll
                        for (int i = 0; i < LD; ++i) acc[j + i] += t[i];
                    }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&ctl.sum_empty));
            }
            if (!ok || !__all_sync(0xffffffffu, gs_wait(smem_u32(&ctl.low_full), (p - p_begin) & 1, abort_flag))) { ok = false; break; }
            tc_fence_after();
#pragma unroll
            for (int j = 0; j < CH; j += LD) {
                float t[LD];
                gs_ld<LD>(mine + HB * NT + j, t);
#pragma unroll
                for (int i = 0; i < LD; ++i) acc[j + i] += t[i];
                if (p > p_begin) {               // the parts before
                    gs_ld<LD>(mine + (HB + 1) * NT + j, t);
#pragma unroll
                    for (int i = 0; i < LD; ++i) acc[j + i] = t[i] + acc[j + i];
                }
                if (p + 1 < p_end) {
#pragma unroll
                    for (int i = 0; i < LD; i += 8) gs_st8(mine + (HB + 1) * NT + j + i, acc + j + i);
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&ctl.low_empty));
        }
        // every product is through with the planes: the tile, [token][row], takes their place
#pragma unroll
        for (int i = 0; i < CH; ++i)
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(planes + ((half * CH + i) * 128 + quarter * 32 + lane) * 4), "f"(acc[i]) : "memory");
    } else {
        // ---- products: the warp walks along together, so that the operands' places stay in uniform registers, one thread issues ----
        constexpr uint32_t idesc = idesc_bf16(128, NT, false);
        const uint32_t base = __shfl_sync(0xffffffffu, tmem, 0), low = base + HB * NT;
        int group = 0;
        for (int p = p_begin; p < p_end; ++p) {
            const int begin = part_begin(p), end = part_begin(p + 1);
            for (int step = begin; step < end; ++step) {
                const int it = step - first, s = it & 1;
                gs_wait(smem_u32(&ctl.full[s]), (it >> 1) & 1, abort_flag);
                const uint32_t at = planes + s * S::STAGE, xat = at + 3 * W_PLANE;
                const uint64_t wh = smem_desc_sw128(at, 16, 1024), xh = smem_desc_sw128(xat, 16, 1024);
                constexpr uint64_t WP = W_PLANE >> 4, XP = S::X_PLANE >> 4;           // the next plane
#pragma unroll
                for (int k0 = 0; k0 < 4; k0 += HB, ++group) {
                    const bool fresh = step == begin && k0 == 0;
                    gs_wait(smem_u32(&ctl.sum_empty), (group & 1) ^ 1, abort_flag);
                    // the part before has been read
                    if (fresh) gs_wait(smem_u32(&ctl.low_empty), ((p - p_begin) & 1) ^ 1, abort_flag);
                    tc_fence_after();
                    if (gs_elect()) {
#pragma unroll
                        for (int k = k0; k < k0 + HB; ++k) gs_umma(base + (k - k0) * NT, wh + 2 * k, xh + 2 * k, idesc, 0u);   // 32 bytes along the swizzled rows
                        umma_commit(smem_u32(&ctl.sum_full));
#pragma unroll
                        for (int k = k0; k < k0 + HB; ++k) {
                            const uint64_t w = wh + 2 * k, x = xh + 2 * k;
                            gs_umma(low, w + 2 * WP, x, idesc, fresh && k == 0 ? 0u : 1u);
                            gs_umma(low, w, x + 2 * XP, idesc, 1u);
                            gs_umma(low, w + WP, x + XP, idesc, 1u);
                            gs_umma(low, w + WP, x, idesc, 1u);
                            gs_umma(low, w, x + XP, idesc, 1u);
                        }
                        if (k0 + HB == 4) {
                            umma_commit(smem_u32(&ctl.empty[s]));
                            if (step + 1 == end) umma_commit(smem_u32(&ctl.low_full));
                        }
                    }
                    __syncwarp();
                }
            }
        }
    }

    if (*abort_flag) {
        // give products in flight time to land before the tensor memory is given back
        for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (*abort_flag) {                           // (every role is through: the flag is settled and nobody else writes to the planes)
        if (tid == 0 && g.err != nullptr) atomicExch(g.err, 1);
        for (int i = tid; i < NT * 128; i += SPLIT_THREADS) asm volatile("st.shared.b32 [%0], %1;" ::"r"(planes + i * 4), "r"(0x7fffffff) : "memory");
        __syncthreads();                         // the tile holds no number: all of it is made again below
    }
    // before the cluster's barrier: a CTA of another launch may be waiting for it where this cluster's next CTA is to wait for that one's
    if (warp == 16) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(S::COLS) : "memory");
    if (g.ranks > 1) gs_cluster_sync();
    const int tokens = min(NT, g.M - m0);
    const bool words = (g.ldc & 3) == 0 && ((uintptr_t)g.C & 15) == 0;
#pragma unroll 1
    for (int e = rank * SPLIT_THREADS + tid; e < tokens * 32; e += g.ranks * SPLIT_THREADS) {
        const int m = m0 + e / 32, n = n0 + (e % 32) * 4;
        if (n >= g.N) continue;
        const uint32_t at = planes + e * 16;
        float v[4];
        {
            float4 t = gs_ld_cluster(g.ranks > 1 ? map_to_rank(at, 0) : map_to_rank(at, cluster_ctarank()));
            for (int p = 1; p < g.ranks; ++p) {
                const float4 u = gs_ld_cluster(map_to_rank(at, p));
                t.x += u.x;
                t.y += u.y;
                t.z += u.z;
                t.w += u.w;
            }
            v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
        }
        const bool finite[4] = {isfinite(v[0]), isfinite(v[1]), isfinite(v[2]), isfinite(v[3])};
        float4 made = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (!(finite[0] && finite[1] && finite[2] && finite[3])) made = gs_again<4>(g.A + (size_t)m * g.lda, g.W + (size_t)n * g.K, g.K, g.N - n, g.a_words);
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            if (n + x >= g.N) continue;
            v[x] = finite[x] ? v[x] * GS_DOWN : x == 0 ? made.x : x == 1 ? made.y : x == 2 ? made.z : made.w;
            if (g.bias) v[x] += g.bias_dtype == MM_F32 ? ((const float*)g.bias)[n + x] : __bfloat162float(((const __nv_bfloat16*)g.bias)[n + x]);
        }
        float* c = g.C + (size_t)m * g.ldc + n;
        if (words && n + 4 <= g.N) {
            *reinterpret_cast<float4*>(c) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
#pragma unroll
            for (int x = 0; x < 4; ++x)
                if (n + x < g.N) c[x] = v[x];
        }
    }
    if (g.ranks > 1) gs_cluster_sync();          // nobody leaves while its tile is read
}

// ---------------------------------------------------------------------------------------------------------------
// a few tokens
// ---------------------------------------------------------------------------------------------------------------
// The same sums in the same order with mma.sync, whose products of sixteen k give the bits that tcgen05's do: a tile of 16 rows of W needs no
// tensor memory, no planes and no hand-over between warps, and there are enough of them to fill the GPU.  A warp takes one part of k of one tile (eight
// warps: 8 / PARTS tiles) and splits both operands' fragments in registers, DEPTH sixteens of k on their way from memory; the
// parts' results meet in shared memory.  Bound by the chain of dependent products (five per sixteen k) and the first loads' latency.
// Weights from memory, single launches, 4 tokens: 896 x 896 10.3 us (by FMAs in order 10.5), 9,728 x 896 18.8 (20.7), 896 x 4,864 16.4 (24.6), 3,584 x 18,944 71
// (160), 37,888 x 3,584 113 (128); 12 tokens: 9,728 x 896 28.7 (34.8), 896 x 4,864 20.6 (28.8), but 896 x 896 12.3 (10.3).  Fragments loaded straight into registers took half as long again: eight cache lines to an eight-byte load.
constexpr int FEW = 16;                       // tokens

__device__ __forceinline__ void gs_mma(float* c, const uint32_t* a, const uint32_t* b) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// N pairs of numbers as three planes
template <int N>
__device__ __forceinline__ void gs_parts(const float2* v, uint32_t (*out)[N]) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
        float x = v[i].x, y = v[i].y;
        gs_up2(x, y);
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            out[p][i] = gs_round2(x, y);
            gs_rest(x, y, out[p][i]);
        }
    }
}

constexpr int FEW_PITCH = 72;                 // floats per row of 64 k: a half warp's eight-byte reads of four rows meet every bank once

template <int NJ, int PARTS>
__global__ void __launch_bounds__(256, NJ == 1 ? 2 : 1) gemv_split_kernel(const SplitArgs g) {
    constexpr int STAGES = NJ == 1 ? 2 : 3, TILES = 8 / PARTS, T = 8 * NJ;
    extern __shared__ __align__(16) float few_smem[];
    __shared__ float sums[8][T][16];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, row = lane >> 2, t2 = (lane & 3) * 2;
    const int part = warp % PARTS, n0 = blockIdx.x * (16 * TILES), r0 = n0 + warp / PARTS * 16;
    const int steps = (g.K + 63) / 64, begin = part * steps / PARTS, end = (part + 1) * steps / PARTS;
    const int floats = (16 + g.M) * FEW_PITCH;              // of a stage: the tile's rows of W, then the tokens
    float* mine = few_smem + warp * (STAGES * floats);
    const uint32_t base = smem_u32(mine);
    auto fetch = [&](int step) {
        const int k = step * 64 + (lane & 15) * 4, r = lane >> 4;
        const bool k_ok = step < end && k < g.K;
        const uint32_t to = base + ((step - begin) % STAGES * floats + r * FEW_PITCH + (lane & 15) * 4) * 4;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const bool in = k_ok && r0 + r + 2 * e < g.N;
            gs_copy<16>(to + e * (2 * FEW_PITCH * 4), in ? g.W + (size_t)(r0 + r + 2 * e) * g.K + k : g.W, in);
        }
        for (int m = r; m < g.M; m += 2) {
            const float* p = k_ok ? g.A + (size_t)m * g.lda + k : g.A;
            const uint32_t at = to + (16 + m - r) * (FEW_PITCH * 4);
            if (g.a_words) gs_copy<16>(at, p, k_ok);
            else
                for (int x = 0; x < 4; ++x) gs_copy<4>(at + 4 * x, k_ok ? p + x : p, k_ok);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
#pragma unroll
    for (int i = 0; i < STAGES; ++i) fetch(begin + i);
    float acc[NJ][4], low[NJ][4];
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[j][i] = low[j][i] = 0.0f;
    int xrow[NJ];                                           // tokens beyond M: sums that nobody reads
#pragma unroll
    for (int j = 0; j < NJ; ++j) xrow[j] = (16 + min(j * 8 + row, g.M - 1)) * FEW_PITCH + t2;
#pragma unroll 1
    for (int step = begin; step < end; ++step) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 1) : "memory");
        __syncwarp();
        const float* s = mine + (step - begin) % STAGES * floats;
        const float* w = s + row * FEW_PITCH + t2;
#pragma unroll
        for (int k = 0; k < 64; k += 16) {
            const float2 wv[4] = {*reinterpret_cast<const float2*>(w + k), *reinterpret_cast<const float2*>(w + 8 * FEW_PITCH + k),
                                  *reinterpret_cast<const float2*>(w + k + 8), *reinterpret_cast<const float2*>(w + 8 * FEW_PITCH + k + 8)};
            uint32_t a[3][4], b[NJ][3][2];
            gs_parts<4>(wv, a);
            float top[NJ][4];
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                const float2 xv[2] = {*reinterpret_cast<const float2*>(s + xrow[j] + k), *reinterpret_cast<const float2*>(s + xrow[j] + k + 8)};
                gs_parts<2>(xv, b[j]);
#pragma unroll
                for (int i = 0; i < 4; ++i) top[j][i] = 0.0f;
            }
#define GS_EACH(C, PW, PX)         \
    _Pragma("unroll") for (int j = 0; j < NJ; ++j) gs_mma(C[j], a[PW], b[j][PX])
            GS_EACH(top, 0, 0);
            GS_EACH(low, 2, 0);
            GS_EACH(low, 0, 2);
            GS_EACH(low, 1, 1);
            GS_EACH(low, 1, 0);
            GS_EACH(low, 0, 1);
#undef GS_EACH
#pragma unroll
            for (int j = 0; j < NJ; ++j)
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[j][i] += top[j][i];
        }
        __syncwarp();
        fetch(step + STAGES);
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) sums[warp][j * 8 + t2 + (i & 1)][row + (i >> 1) * 8] = acc[j][i] + low[j][i];
    __syncthreads();
    for (int e = threadIdx.x; e < g.M * 16 * TILES; e += 256) {
        const int m = e / (16 * TILES), c = e % (16 * TILES), n = n0 + c;
        if (n >= g.N) continue;
        const int first = c / 16 * PARTS;
        float v = sums[first][m][c % 16];
#pragma unroll
        for (int p = 1; p < PARTS; ++p) v += sums[first + p][m][c % 16];
        if (isfinite(v)) v *= GS_DOWN;
        else v = gs_again<1>(g.A + (size_t)m * g.lda, g.W + (size_t)n * g.K, g.K, 1, g.a_words).x;
        if (g.bias) v += g.bias_dtype == MM_F32 ? ((const float*)g.bias)[n] : __bfloat162float(((const __nv_bfloat16*)g.bias)[n]);
        g.C[(size_t)m * g.ldc + n] = v;
    }
}

template <int NJ, int PARTS>
int launch_few(const SplitArgs& g, cudaStream_t s) {
    constexpr int stages = NJ == 1 ? 2 : 3;
    if (!mm_allow_smem<gemv_split_kernel<NJ, PARTS>>(8 * stages * (16 + 8 * NJ) * FEW_PITCH * 4)) {
        mm_set_last_error("gemm: cannot reserve shared memory");
        return MM_ERR_LAUNCH;
    }
    mm_launch(gemv_split_kernel<NJ, PARTS>, dim3(ceil_div(g.N, 16 * (8 / PARTS))), dim3(256), (size_t)(8 * stages * (16 + g.M) * FEW_PITCH * 4), s, g);
    MM_CHECK_LAUNCH();
    return MM_OK;
}
template <int NJ>
int launch_few(const SplitArgs& g, cudaStream_t s) {
    switch (g.parts) {
        case 1: return launch_few<NJ, 1>(g, s);
        case 2: return launch_few<NJ, 2>(g, s);
        case 4: return launch_few<NJ, 4>(g, s);
        default: return launch_few<NJ, 8>(g, s);
    }
}

// k in parts: eight of at least four steps of 64, or as many as there are
int gemm_split_parts(int K) {
    const int steps = ceil_div(K, 64);
    return steps >= 24 ? 8 : steps >= 10 ? 4 : steps >= 4 ? 2 : 1;
}

SplitArgs split_args(const float* A, const float* W, const void* bias, int bias_dtype, float* C, int M, int N, int K, int lda, int ldc, int* err, int give_up) {
    return SplitArgs{A, W, bias, C, bias_dtype, M, N, K, lda, ldc, gemm_split_parts(K), 1, lda % 4 == 0 && ((uintptr_t)A & 15) == 0, err, give_up};
}

template <int NT>
int launch_split(SplitArgs g, int ranks, cudaStream_t s) {
    g.ranks = ranks;
    if (!mm_allow_smem<gemm_split_kernel<NT>>(SplitShape<NT>::SMEM)) {
        mm_set_last_error("gemm: cannot reserve shared memory");
        return MM_ERR_LAUNCH;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ranks * ceil_div(g.M, NT), ceil_div(g.N, 128));
    cfg.blockDim = dim3(SPLIT_THREADS);
    cfg.dynamicSmemBytes = SplitShape<NT>::SMEM;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ranks;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, gemm_split_kernel<NT>, g);
    MM_CHECK_LAUNCH();
    return MM_OK;
}

int launch_split(const SplitArgs& g, int nt, int ranks, cudaStream_t s) {
    switch (nt) {
        case FEW: return g.M <= 8 ? launch_few<1>(g, s) : launch_few<2>(g, s);
        case 32: return launch_split<32>(g, ranks, s);
        case 64: return launch_split<64>(g, ranks, s);
        default: return launch_split<128>(g, ranks, s);
    }
}

}  // namespace

static bool gemm_split_can(const void* W, int K) { return K % 4 == 0 && ((uintptr_t)W & 15) == 0; }

// By the weights alone, never by M.  Not the products whose weights are mostly streamed, a head's 151,936 rows: there a few tokens' sums by FMAs
// read them faster (545 MB for 4 tokens 121 us from memory, 127 here), and many tokens are rare.  Nor small weights, where the fixed costs of the split decide for
// a few tokens, which is what most steps have, and prompts gain little.  us for 1, 4, 8, 64 and 1,024 tokens, weights from memory, by FMAs and here:
//   512 x 256     2.8  2.9  2.9  11  11      3.8  4.1  4.3  7.7  10        4,864 x 256   3.7  4.6  5.6  12   67      4.5  4.8  5.1  9.6  42
//   1,024 x 512   3.8  4.2  4.4  22  30      5.8  6.2  6.4  9.8  15        9,728 x 128   3.3  5.1  5.8  9.5  62      4.6  5.5  6.0  8.7  49
//   2,048 x 512   4.3  5.2  5.8  22  58      6.0  6.3  6.7  10   22        128 x 640     3.7  3.9  4.0  22   24      4.6  4.8  5.2  8.6  9.1
//   1,024 x 896   5.2  5.7  6.0  38  50      5.9  6.1  6.4  10   25        128 x 2,048   8.5  8.9  9.4  70   78      5.6  5.9  6.2  10   16
// So k of ten steps and more, which go in four or eight parts, or 1.2 million numbers: a few tokens lose a quarter at the most there, many take half
// as long or less.
bool gemm_split_takes(const void* W, int N, int K) {
    return gemm_split_can(W, K) && N >= 128 && N <= 65536 && K >= 128 && (K > 9 * 64 || (long long)N * K >= 1200000);
}

int gemm_split(const float* A, const float* W, const void* bias, int bias_dtype, float* C, int M, int N, int K, int lda, int ldc, int* err,
               cudaStream_t s) {
    const SplitArgs g = split_args(A, W, bias, bias_dtype, C, M, N, K, lda, ldc, err, 0);
    if (M <= FEW) return launch_split(g, FEW, 1, s);
    // The tile and the parts' place that take the least time: rounds of one CTA per SM (clusters of 4 find room for 132 CTAs, of 8 for 120), each with a start (8 us with the first loads and the end) and
    // a time per 64 k that was measured for each tile, and 2 us where a cluster's results meet.  Within 15 % of what is measured
    // for 17 to 1,024 tokens of 896 to 9,728 rows.
    constexpr int TILES[3] = {32, 64, 128}, STEP_NS[3] = {1030, 1220, 1700};
    const int steps = ceil_div(K, 64);
    long long best = -1;
    int nt = 32, ranks = 1;
    for (int i = 0; i < 3; ++i) {
        for (const int r : {1, g.parts}) {
            const long long ctas = (long long)ceil_div(M, TILES[i]) * ceil_div(N, 128) * r;
            const int room = r == 8 ? 120 : r == 4 ? 132 : 148;
            const long long ns = (ctas + room - 1) / room * (8000 + (long long)ceil_div(steps, r) * STEP_NS[i]) + (r > 1 ? 2000 : 0);
            if (best < 0 || ns < best) {
                best = ns;
                nt = TILES[i];
                ranks = r;
            }
        }
    }
    return launch_split(g, nt, ranks, s);
}

// The same product in a form of the caller's choice, which does not change a bit: tiles of `tile` tokens (16: the kernel for up to
// so many; 32, 64 or 128), the parts of k one after the other or in a cluster.  `give_up`: 1 as if a wait of the tiles' kernel had run out at its
// start.
MM_EXPORT int mm_gemm_split(const void* A, const void* W, const void* bias, int bias_dtype, void* C, int M, int N, int K, int lda, int ldc, int tile,
                            int side_by_side, int give_up, void* err, void* stream) {
    MM_REQUIRE(M > 0 && N > 0 && K > 0 && lda >= K && ldc >= N && gemm_split_can(W, K), "gemm_split: bad sizes");
    MM_REQUIRE((tile == FEW && M <= FEW) || tile == 32 || tile == 64 || tile == 128, "gemm_split: no such tile");
    const SplitArgs g = split_args((const float*)A, (const float*)W, bias, bias_dtype, (float*)C, M, N, K, lda, ldc, (int*)err, give_up);
    return launch_split(g, tile, side_by_side ? g.parts : 1, (cudaStream_t)stream);
}
