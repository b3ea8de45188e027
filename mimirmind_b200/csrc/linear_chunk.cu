// The matrix-state recurrence (csrc/linear_state.cu) over long portions as products of matrices, 64 tokens at a time.
//
// Within a chunk, with gamma_t the product of the decays up to token t and S the state before it ([dk, dv]),
//
//   o_t = gamma_t S^T q_t + sum_(s <= t) (gamma_t / gamma_s) (q_t . k_s) u_s,      S' = gamma_C S + sum_s (gamma_C / gamma_s) k_s u_s^T,
//
// where u = v without the delta rule.  With it, u = beta (v - g S^T k) is the solution of a unit triangular system,
//
//   (I + L) U = diag(beta) (V - diag(gamma) K S),      L[t, s] = beta_t (gamma_t / gamma_s) (k_t . k_s) for s < t,
//
// so with T = (I + L)^-1, W = T diag(beta gamma) K and U0 = T diag(beta) V it is U = U0 - W S: only that product and S' have to
// wait for the chunk before (the WY form of a product of rank-one updates, Bischof and Van Loan 1987).  The launches:
//   plain:  lc_state (what each chunk adds), lc_carry over the chunks per number of the state, lc_output;
//   delta:  lc_delta_prepare (T, W, U0 per chunk), lc_delta_carry (U and S', chunk after chunk), lc_output with u for v.
// A token costs dk dv multiply-adds three to four times as in the token-by-token walk, but as tiles of 16 x 8 x 16 on the tensor
// cores (mma.sync): every operand is split into three bf16 numbers, which hold all of its 24 bits (of numbers below 2^-110 fewer: bf16 ends at
// 2^-133), and the product is the sum of the six larger of the nine partial products, added up in 32 bits (Henry, Tang and Heinecke 2019).  Error against 64 bits, of outputs and states over 300 to 4,096 tokens: where many tokens
// add up (decays near 1) 0.7e-7 to 1.4e-7, half of the 32-bit walk's; where a state forgets half of itself per token, so that the
// walk has little left to round, 0.6e-7 to 1.2e-7 (the walk: 0.4e-7 to 0.9e-7).  With two tf32 numbers (22 bits) and three products it was
// 1.0e-7 to 2.4e-7 in both, for kernels 5 to 8 % shorter.  The FMA units, whose tiles are held up by shared-memory reads, take twice as long.
// Ratios of decays are exponentials of differences of the logarithms' sums, which are kept in 64 bits: quotients of products of
// the decays themselves would underflow within a chunk (0.2 a token), differences of 32-bit sums lose what lies close together.
#include "common.cuh"

#include <type_traits>

#define LC_C 64              // tokens per chunk
#define LC_LD 136            // floats per row of a [tokens, 128] tile: rows 8 banks apart
#define LC_LP 68             // floats per row of a [64, 64] tile that is read along its rows: rows 4 banks apart

__device__ __forceinline__ void lc_cp16(void* smem, const void* gmem, bool in) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(smem);
    const int bytes = in ? 16 : 0;               // 0: zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(gmem), "r"(bytes));
}
__device__ __forceinline__ void lc_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void lc_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// rows [0, 64) x columns [0, COLS) of a matrix of `rows` x `cols` numbers (row stride ld) into shared memory, zeros beyond
template <int COLS, int LD, int THREADS = 256>
__device__ __forceinline__ void lc_load(float* s, const float* __restrict__ p, size_t ld, int rows, int cols) {
    constexpr int Q = COLS / 4;
#pragma unroll
    for (int e = 0; e < 64 * Q / THREADS; ++e) {
        const int idx = threadIdx.x + e * THREADS, r = idx / Q, c = (idx % Q) * 4;
        const bool in = r < rows && c < cols;
        lc_cp16(s + r * LD + c, p + (in ? (size_t)r * ld + c : 0), in);
    }
}

// Whether the 16-byte pieces that this thread itself has brought in with lc_load (and waited for) hold a number that the products turn into a NaN:
// a NaN, an infinity or one beyond bf16's range.
template <int COLS, int LD, int THREADS = 256>
__device__ __forceinline__ bool lc_not_finite(const float* s) {
    constexpr int Q = COLS / 4;
    uint32_t top = 0;
#pragma unroll
    for (int e = 0; e < 64 * Q / THREADS; ++e) {
        const int idx = threadIdx.x + e * THREADS;
        const uint4 v = *reinterpret_cast<const uint4*>(s + (idx / Q) * LD + (idx % Q) * 4);
        top = max(max(max(v.x & 0x7fffffffu, v.y & 0x7fffffffu), max(v.z & 0x7fffffffu, v.w & 0x7fffffffu)), top);
    }
    return top >= 0x7f7f8000u;
}

// Two numbers as three bf16 pairs each, x = h + m + l: every part is the rest rounded to 8 bits, so the three hold all 24 bits of x
// (from 3.4e38, bf16's largest number, on x counts as infinite).
struct LcSplit {
    uint32_t h, m, l;
};
__device__ __forceinline__ uint32_t lc_round2(float x, float y) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(y), "f"(x));
    return r;
}
__device__ __forceinline__ LcSplit lc_split(float x, float y) {
    LcSplit r;
    r.h = lc_round2(x, y);
    x = __fsub_rn(x, __uint_as_float(r.h << 16));
    y = __fsub_rn(y, __uint_as_float(r.h & 0xffff0000u));
    r.m = lc_round2(x, y);
    x = __fsub_rn(x, __uint_as_float(r.m << 16));
    y = __fsub_rn(y, __uint_as_float(r.m & 0xffff0000u));
    r.l = lc_round2(x, y);
    return r;
}
// The same of x f and y e, whose roundings go into the last parts.
__device__ __forceinline__ LcSplit lc_split(float x, float f, float y, float e) {
    const float p = __fmul_rn(x, f), q = __fmul_rn(y, e);
    const float dp = __fmaf_rn(x, f, -p), dq = __fmaf_rn(y, e, -q);
    LcSplit r;
    r.h = lc_round2(p, q);
    x = __fsub_rn(p, __uint_as_float(r.h << 16));
    y = __fsub_rn(q, __uint_as_float(r.h & 0xffff0000u));
    r.m = lc_round2(x, y);
    x = __fadd_rn(__fsub_rn(x, __uint_as_float(r.m << 16)), dp);
    y = __fadd_rn(__fsub_rn(y, __uint_as_float(r.m & 0xffff0000u)), dq);
    r.l = lc_round2(x, y);
    return r;
}
struct LcA {
    LcSplit x[4];
};
struct LcB {
    LcSplit x[2];
};
__device__ __forceinline__ void lc_mma(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void lc_mma_first(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
        : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.0f));
}
__device__ __forceinline__ void lc_mma_half(float* c, uint32_t a0, uint32_t a1, uint32_t b0) {      // eight k, from zero
    asm("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};\n"
        : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
        : "r"(a0), "r"(a1), "r"(b0), "f"(0.0f));
}
// acc[i][j] += the largest partial products of A_i B_j over sixteen k, low[i][j] += the next five (the three below 2^-25 of the whole are left out).
// The tensor core shifts the products of a sum to the place of the largest and cuts off what falls below 2^-24 of it instead of rounding, so a
// chain of sums of full 24-bit numbers drifts.  The largest products have 16 bits each: sixteen of them, from zero, lose little, and
// the FMA units, which round to nearest, add that on.  What is cut off the others, 2^-8 of them, is as much smaller, so they
// stay on the tensor core for all of k.  The result is acc + low: one rounding, where a chain of FMAs has one per k.  The steps go over
// all tiles in turn: one tile's next step would wait for its last.
// EIGHT: the largest products eight k at a time, for sums whose terms span many binades (the forget gate's states are off by 5.3e-8 of them so
// instead of 6.3e-8; 2,048 tokens in 20.4 us instead of 19.5; elsewhere it costs 4 to 11 % and gains something only under strong decays).
template <int NI, int NJ, bool EIGHT = false>
__device__ __forceinline__ void lc_products(float (*acc)[NJ][4], float (*low)[NJ][4], const LcA* a, const LcB* b) {
    constexpr int PARTS = EIGHT ? 2 : 1;
    float t[PARTS][NI][NJ][4];
#define LC_TILES                                   \
    _Pragma("unroll") for (int j = 0; j < NJ; ++j) \
    _Pragma("unroll") for (int i = 0; i < NI; ++i)
#define LC_PART(MMA, TO, PA, PB) \
    LC_TILES MMA(TO[i][j], a[i].x[0].PA, a[i].x[1].PA, a[i].x[2].PA, a[i].x[3].PA, b[j].x[0].PB, b[j].x[1].PB)
    if constexpr (EIGHT) {
#pragma unroll
        for (int p = 0; p < PARTS; ++p) LC_TILES lc_mma_half(t[p][i][j], a[i].x[2 * p].h, a[i].x[2 * p + 1].h, b[j].x[p].h);
    } else {
        LC_PART(lc_mma_first, t[0], h, h);
    }
    LC_PART(lc_mma, low, l, h);
    LC_PART(lc_mma, low, h, l);
    LC_PART(lc_mma, low, m, m);
    LC_PART(lc_mma, low, m, h);
    LC_PART(lc_mma, low, h, m);
#pragma unroll
    for (int p = 0; p < PARTS; ++p)
        LC_TILES
#pragma unroll
        for (int x = 0; x < 4; ++x) acc[i][j][x] += t[p][i][j][x];
#undef LC_PART
#undef LC_TILES
}
// The same for one column tile and 32 rows, acc[16 rows].
template <bool EIGHT = false>
__device__ __forceinline__ void lc_one(float (*acc)[4], float (*low)[4], const LcA* a, const LcB& b) {
    lc_products<2, 1, EIGHT>(reinterpret_cast<float(*)[1][4]>(acc), reinterpret_cast<float(*)[1][4]>(low), a, &b);
}
template <int N>
__device__ __forceinline__ void lc_zero(float* v) {
#pragma unroll
    for (int x = 0; x < N; ++x) v[x] = 0.0f;
}
template <int N>
__device__ __forceinline__ void lc_add(float* v, const float* w) {
#pragma unroll
    for (int x = 0; x < N; ++x) v[x] += w[x];
}
// Fragments of sixteen k.  "rows": the operand stands as [m or n][k]; a thread takes k 2t, 2t + 1, 2t + 8 and 2t + 9 for its four places (any order
// of k will do, as long as both operands have the same), as two 8-byte words.  "rows4": the same in the order t, t + 4, t + 8, t + 12, for a
// product whose other operand stands as [k][n].  "cols": the operand stands as [k][m or n], order t, t + 4, t + 8, t + 12.
__device__ __forceinline__ float2 lc_pair(const float* p) { return *reinterpret_cast<const float2*>(p); }
__device__ __forceinline__ LcA lc_a_rows(const float* p, int ld) {
    const int g = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
    const float* lo = p + g * ld + 2 * t;
    const float* hi = lo + 8 * ld;
    const float2 w = lc_pair(lo), x = lc_pair(hi), y = lc_pair(lo + 8), z = lc_pair(hi + 8);
    return LcA{{lc_split(w.x, w.y), lc_split(x.x, x.y), lc_split(y.x, y.y), lc_split(z.x, z.y)}};
}
// "rows" with a factor per k: scale points at the first of the sixteen
__device__ __forceinline__ LcA lc_a_rows_scaled(const float* p, int ld, const float* scale) {
    const int g = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
    const float* lo = p + g * ld + 2 * t;
    const float* hi = lo + 8 * ld;
    const float2 w = lc_pair(lo), x = lc_pair(hi), y = lc_pair(lo + 8), z = lc_pair(hi + 8);
    const float2 f = lc_pair(scale + 2 * t), e = lc_pair(scale + 2 * t + 8);
    return LcA{{lc_split(w.x, f.x, w.y, f.y), lc_split(x.x, f.x, x.y, f.y), lc_split(y.x, e.x, y.y, e.y), lc_split(z.x, e.x, z.y, e.y)}};
}
__device__ __forceinline__ LcB lc_b_rows(const float* p, int ld) {
    const int g = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
    const float2 x = lc_pair(p + g * ld + 2 * t), y = lc_pair(p + g * ld + 2 * t + 8);
    return LcB{{lc_split(x.x, x.y), lc_split(y.x, y.y)}};
}
// the factors of a thread's four k: scale points at the first of the sixteen
struct LcScale {
    float f[4];
};
__device__ __forceinline__ LcScale lc_scale(const float* scale) {
    const int t = threadIdx.x & 3;
    return LcScale{{scale[t], scale[t + 4], scale[t + 8], scale[t + 12]}};
}
__device__ __forceinline__ LcA lc_a_rows4(const float* p, int ld) {
    const int g = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
    const float* lo = p + g * ld + t;
    const float* hi = lo + 8 * ld;
    return LcA{{lc_split(lo[0], lo[4]), lc_split(hi[0], hi[4]), lc_split(lo[8], lo[12]), lc_split(hi[8], hi[12])}};
}
__device__ __forceinline__ LcA lc_a_rows4(const float* p, int ld, const LcScale& s) {
    const int g = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
    const float* lo = p + g * ld + t;
    const float* hi = lo + 8 * ld;
    return LcA{{lc_split(lo[0], s.f[0], lo[4], s.f[1]), lc_split(hi[0], s.f[0], hi[4], s.f[1]), lc_split(lo[8], s.f[2], lo[12], s.f[3]),
                lc_split(hi[8], s.f[2], hi[12], s.f[3])}};
}
__device__ __forceinline__ LcA lc_a_cols(const float* p, int ld, const LcScale& s) {
    const int g = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
    const float* q = p + t * ld + g;
    return LcA{{lc_split(q[0], s.f[0], q[4 * ld], s.f[1]), lc_split(q[8], s.f[0], q[4 * ld + 8], s.f[1]),
                lc_split(q[8 * ld], s.f[2], q[12 * ld], s.f[3]), lc_split(q[8 * ld + 8], s.f[2], q[12 * ld + 8], s.f[3])}};
}
__device__ __forceinline__ LcB lc_b_cols(const float* p, int ld) {
    const int g = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
    const float* q = p + t * ld + g;
    return LcB{{lc_split(q[0], q[4 * ld]), lc_split(q[8 * ld], q[12 * ld])}};
}

// ---- operands split once, by the block: three planes of bf16 in shared memory --------------------------------------------------
// A tile [rows][COLS] as its parts h, m and l, each [rows][COLS + 8] in bf16: rows 16 bytes off a multiple of 128, so that ldmatrix, which
// reads eight rows' 16 bytes, meets every bank once.  Split while it is brought in, an operand costs its eleven instructions per two
// numbers once and not in every warp that multiplies with it.
template <int COLS>
__host__ __device__ constexpr int lc_plane(int rows) { return rows * (COLS + 8) * 2; }        // bytes of one of the three
__device__ __forceinline__ void lc_sts64(uint32_t to, uint32_t x, uint32_t y) { asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(to), "r"(x), "r"(y) : "memory"); }
__device__ __forceinline__ void lc_sts32(uint32_t to, uint32_t x) { asm volatile("st.shared.b32 [%0], %1;" ::"r"(to), "r"(x) : "memory"); }
__device__ __forceinline__ void lc_put4(uint32_t to, int plane, const LcSplit& x, const LcSplit& y) {
    lc_sts64(to, x.h, y.h);
    lc_sts64(to + plane, x.m, y.m);
    lc_sts64(to + 2 * plane, x.l, y.l);
}
__device__ __forceinline__ uint32_t lc_top(const float4& v) {             // (see lc_not_finite)
    const uint32_t a = __float_as_uint(v.x) & 0x7fffffffu, b = __float_as_uint(v.y) & 0x7fffffffu, c = __float_as_uint(v.z) & 0x7fffffffu,
                   d = __float_as_uint(v.w) & 0x7fffffffu;
    return max(max(a, b), max(c, d));
}
// A thread's 16-byte pieces of rows [0, 64) x columns [0, COLS) of a matrix of `rows` x `cols` numbers, zeros beyond; and these as planes.
template <int COLS>
struct LcTile {
    static constexpr int Q = COLS / 4, N = 64 * Q / 256;
    float4 v[N];
    __device__ __forceinline__ void load(const float* __restrict__ p, size_t ld, int rows, int cols) {
#pragma unroll
        for (int e = 0; e < N; ++e) {
            const int idx = threadIdx.x + e * 256, r = idx / Q, c = (idx % Q) * 4;
            v[e] = r < rows && c < cols ? __ldg(reinterpret_cast<const float4*>(p + (size_t)r * ld + c)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    }
    __device__ __forceinline__ void to_planes(uint32_t planes) const {
#pragma unroll
        for (int e = 0; e < N; ++e) {
            const int idx = threadIdx.x + e * 256, r = idx / Q, c = (idx % Q) * 4;
            lc_put4(planes + (r * (COLS + 8) + c) * 2, lc_plane<COLS>(64), lc_split(v[e].x, v[e].y), lc_split(v[e].z, v[e].w));
        }
    }
    __device__ __forceinline__ void to_floats(float* s) const {            // [64][LC_LD]
#pragma unroll
        for (int e = 0; e < N; ++e) {
            const int idx = threadIdx.x + e * 256;
            *reinterpret_cast<float4*>(s + (idx / Q) * LC_LD + (idx % Q) * 4) = v[e];
        }
    }
    __device__ __forceinline__ bool not_finite() const {
        uint32_t top = 0u;
#pragma unroll
        for (int e = 0; e < N; ++e) top = max(top, lc_top(v[e]));
        return top >= 0x7f7f8000u;
    }
};
__device__ __forceinline__ void lc_ldsm(uint32_t at, uint32_t& a, uint32_t& b, uint32_t& c, uint32_t& d) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(a), "=r"(b), "=r"(c), "=r"(d) : "r"(at) : "memory");
}
__device__ __forceinline__ void lc_ldsm_t(uint32_t at, uint32_t& a, uint32_t& b, uint32_t& c, uint32_t& d) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(a), "=r"(b), "=r"(c), "=r"(d) : "r"(at) : "memory");
}
// Fragments of sixteen k from planes with rows of LD numbers; `at` is the address of the sub-tile's first number in plane h.
// a_mk: the operand stands as [m][k]; a_km: as [k][m]; b2_nk and b2_kn: two tiles of eight columns, [n][k] and [k][n].
template <int LD>
__device__ __forceinline__ LcA lc_a_mk(uint32_t at, int plane) {
    const int lane = threadIdx.x & 31;
    at += (((lane & 7) + (lane & 8)) * LD + (lane & 16) / 2) * 2;
    LcA r;
    lc_ldsm(at, r.x[0].h, r.x[1].h, r.x[2].h, r.x[3].h);
    lc_ldsm(at + plane, r.x[0].m, r.x[1].m, r.x[2].m, r.x[3].m);
    lc_ldsm(at + 2 * plane, r.x[0].l, r.x[1].l, r.x[2].l, r.x[3].l);
    return r;
}
template <int LD>
__device__ __forceinline__ LcA lc_a_km(uint32_t at, int plane) {
    const int lane = threadIdx.x & 31;
    at += (((lane & 7) + (lane & 16) / 2) * LD + (lane & 8)) * 2;
    LcA r;
    lc_ldsm_t(at, r.x[0].h, r.x[1].h, r.x[2].h, r.x[3].h);
    lc_ldsm_t(at + plane, r.x[0].m, r.x[1].m, r.x[2].m, r.x[3].m);
    lc_ldsm_t(at + 2 * plane, r.x[0].l, r.x[1].l, r.x[2].l, r.x[3].l);
    return r;
}
template <int LD>
__device__ __forceinline__ void lc_b2_nk(uint32_t at, int plane, LcB* b) {
    const int lane = threadIdx.x & 31;
    at += (((lane & 7) + (lane & 16) / 2) * LD + (lane & 8)) * 2;
    lc_ldsm(at, b[0].x[0].h, b[0].x[1].h, b[1].x[0].h, b[1].x[1].h);
    lc_ldsm(at + plane, b[0].x[0].m, b[0].x[1].m, b[1].x[0].m, b[1].x[1].m);
    lc_ldsm(at + 2 * plane, b[0].x[0].l, b[0].x[1].l, b[1].x[0].l, b[1].x[1].l);
}
template <int LD>
__device__ __forceinline__ void lc_b2_kn(uint32_t at, int plane, LcB* b) {
    const int lane = threadIdx.x & 31;
    at += (((lane & 7) + (lane & 8)) * LD + (lane & 16) / 2) * 2;
    lc_ldsm_t(at, b[0].x[0].h, b[0].x[1].h, b[1].x[0].h, b[1].x[1].h);
    lc_ldsm_t(at + plane, b[0].x[0].m, b[0].x[1].m, b[1].x[0].m, b[1].x[1].m);
    lc_ldsm_t(at + 2 * plane, b[0].x[0].l, b[0].x[1].l, b[1].x[0].l, b[1].x[1].l);
}

// The sums of the decays' logarithms over the chunk's tokens, sb[t] = log gamma_t, by the first two warps; tokens beyond the
// chunk add nothing.  A decay of 0 counts as exp(-200), which no 32-bit number can tell from it; one that is no number (or negative) is
// NaN here, and so is all that comes after it.
__device__ __forceinline__ void lc_decays(const float* __restrict__ gate, const float* __restrict__ head_decay, int t0, int cnt, int H, int h,
                                          double* sb) {
    __shared__ double first_half;
    double x = 0.0;
    const int t = threadIdx.x, lane = t & 31;
    if (t < LC_C) {
        if (t < cnt) {
            const float l = logf(gate ? gate[(size_t)(t0 + t) * H + h] : head_decay[h]);
            x = (double)(l < -200.0f ? -200.0f : l);         // (keeps a NaN, which fmaxf would not)
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double up = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += up;
        }
        if (t == 31) first_half = x;
    }
    __syncthreads();
    if (t < LC_C) sb[t] = t >= 32 ? x + first_half : x;
    __syncthreads();
}
__device__ __forceinline__ float lc_exp(double x) { return expf((float)x); }

// acc += scores [64][LC_LP] x values [64][LC_LD] for the warp's rows m0.. and columns, a row's own token and those before it only: a product of tiles
// multiplies a later token's numbers with zeros, and where they are infinite or NaN that is a NaN.  Taken by chunks that hold such
// a number, whose outputs before its token stay what they are without it.
__device__ __noinline__ float lc_causal_sum(float sum, const float* scores, const float* values, int m) {
    for (int s = 0; s <= m; ++s) sum = fmaf(scores[s], values[s * LC_LD], sum);
    return sum;
}
// acc [16 rows][8 columns] of a warp's 32 rows and sixteen columns
__device__ __forceinline__ void lc_causal(float (*acc)[2][4], const float* scores, const float* values, int m0, int wn) {
    const int t = threadIdx.x & 3, g = (threadIdx.x & 31) >> 2;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const int m = m0 + 16 * i + g + 8 * (x >> 1), n = wn * 16 + 8 * j + 2 * t + (x & 1);
                acc[i][j][x] = lc_causal_sum(acc[i][j][x], scores + m * LC_LP, values + n, m);
            }
}

__device__ __forceinline__ void lc_causal_cols(float (*acc)[2][4], const float* scores, const float* values, int m0, int wn) {     // acc [8 columns][16 rows]
    float r[2][2][4];
#pragma unroll
    for (int x = 0; x < 16; ++x) r[(x >> 2) & 1][x >> 3][x & 3] = acc[x >> 3][(x >> 2) & 1][x & 3];
    lc_causal(r, scores, values, m0, wn);
#pragma unroll
    for (int x = 0; x < 16; ++x) acc[x >> 3][(x >> 2) & 1][x & 3] = r[(x >> 2) & 1][x >> 3][x & 3];
}

struct LcArgs {
    const float *q, *k, *v, *gate, *beta, *head_decay;
    int ldq, ldk, ldv;
    float *out, *state;
    long long state_stride;
    const int32_t *chunk_meta, *req_chunks, *slots, *positions;
    int n_chunks, H, G, dk, dv;
    float *states;       // [chunks, H, dv, dk]: what a chunk adds, then what it starts from
    float *gain;         // [chunks, H]: gamma_C
    uint4* frag;         // fragments of W and of K' per chunk and head (delta rule, see lc_delta_prepare_kernel)
    float* u;            // [tokens, H dv] (delta rule)
};

// V^T diag(sr) K of a chunk, [dv, dk], to its place in `states`; k and v stand in shared memory.
template <int DK, int DV, bool EIGHT = false>
__device__ __forceinline__ void lc_add_up(const LcArgs& a, int h, int c, const float* sk, const float* sv, const float* sr) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int WM = DV / 32, WN = 8 / WM, NT = DK / WN / 8;      // warps along dv (32 rows each) and dk; tiles of 8 columns per warp
    constexpr int RUN = NT < 4 ? NT : 4;         // column tiles at a time: more would not fit the registers
    const int m0 = (warp % WM) * 32, n0 = (warp / WM) * (DK / WN);
    const int t = lane & 3, g = lane >> 2;
    float* o = a.states + ((size_t)c * a.H + h) * a.dv * a.dk;
#pragma unroll 1
    for (int j0 = 0; j0 < NT; j0 += RUN) {
        float acc[RUN][2][1][4], low[RUN][2][1][4];      // [column tile][16 rows]
        lc_zero<RUN * 8>(&acc[0][0][0][0]);
        lc_zero<RUN * 8>(&low[0][0][0][0]);
#pragma unroll 1
        for (int k0 = 0; k0 < LC_C; k0 += 16) {
            const LcScale scale = lc_scale(sr + k0);
            LcA fa[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) fa[i] = lc_a_cols(sv + k0 * LC_LD + m0 + 16 * i, LC_LD, scale);
#pragma unroll
            for (int j = 0; j < RUN; ++j) {
                const LcB fb = lc_b_cols(sk + k0 * LC_LD + n0 + 8 * (j0 + j), LC_LD);
                lc_products<2, 1, EIGHT>(acc[j], low[j], fa, &fb);
            }
        }
        lc_add<RUN * 8>(&acc[0][0][0][0], &low[0][0][0][0]);
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < RUN; ++j) {
                const int n = n0 + 8 * (j0 + j) + 2 * t;
                if (n >= a.dk) continue;
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const int m = m0 + 16 * i + g + 8 * half;
                    if (m < a.dv) *reinterpret_cast<float2*>(o + (size_t)m * a.dk + n) = make_float2(acc[j][i][0][2 * half], acc[j][i][0][2 * half + 1]);
                }
            }
    }
}

// ---- what a chunk adds to the state, as [dv, dk]: V^T diag(gamma_C / gamma) K -------------------------------------------------
// Bound by the tensor cores and, with 64 KB of result per 64 tokens and head, by writing it.
template <int DK, int DV>
__global__ void __launch_bounds__(256, 2) lc_state_kernel(LcArgs a) {
    extern __shared__ __align__(16) float lc_smem[];
    float* sk = lc_smem;                         // [64][LC_LD]
    float* sv = sk + LC_C * LC_LD;               // [64][LC_LD]
    __shared__ double sb[LC_C];
    __shared__ float sr[LC_C];
    const int h = blockIdx.x, c = blockIdx.y;
    const int t0 = a.chunk_meta[4 * c], cnt = a.chunk_meta[4 * c + 1];
    const int kh = h / (a.H / a.G);
    lc_load<DK, LC_LD>(sk, a.k + (size_t)t0 * a.ldk + (size_t)kh * a.dk, a.ldk, cnt, a.dk);
    lc_load<DV, LC_LD>(sv, a.v + (size_t)t0 * a.ldv + (size_t)h * a.dv, a.ldv, cnt, a.dv);
    lc_commit();
    lc_decays(a.gate, a.head_decay, t0, cnt, a.H, h, sb);
    if (threadIdx.x < LC_C) sr[threadIdx.x] = lc_exp(sb[LC_C - 1] - sb[threadIdx.x]);
    if (threadIdx.x == 0) a.gain[(size_t)c * a.H + h] = lc_exp(sb[LC_C - 1]);
    lc_wait<0>();
    __syncthreads();
    lc_add_up<DK, DV>(a, h, c, sk, sv, sr);
}

// The carry over the chunks, a thread per four numbers of the state: gain [chunks, H], or with a factor per key channel [chunks, H, dk].
// Bound by memory; 48 states of 2 MB, more than L2 holds beside what it still writes back: 44 us (eight loads, then their eight sums, then the next: 80).
template <bool CHANNEL>
__global__ void __launch_bounds__(256) lc_carry_kernel(LcArgs a) {
    const long long size = (long long)a.H * a.dv * a.dk, i = 4 * ((long long)blockIdx.x * 256 + threadIdx.x);
    const int r = blockIdx.y;
    if (i >= size) return;
    const int h = (int)(i / (a.dv * a.dk)), first = a.req_chunks[2 * r], count = a.req_chunks[2 * r + 1];
    if (count <= 0) return;
    float* base = a.states + (size_t)first * size + i;
    const float* gain = a.gain + (CHANNEL ? ((size_t)first * a.H + h) * a.dk + i % a.dk : (size_t)first * a.H + h);
    const int step = CHANNEL ? a.H * a.dk : a.H;
    float* st = a.state + (size_t)a.slots[r] * a.state_stride + i;
    const bool fresh = a.positions[a.chunk_meta[4 * first]] == 0;
    float4 S = fresh ? make_float4(0.0f, 0.0f, 0.0f, 0.0f) : make_float4(st[0], st[1], st[2], st[3]);
    if constexpr (CHANNEL) {
        for (int c0 = 0; c0 < count; c0 += 8) {      // (8 us for 32 chunks of 16 states of 128 x 64; the loop below 11)
            float4 add[8], g[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const bool in = c0 + j < count;
                add[j] = in ? *reinterpret_cast<const float4*>(base + (size_t)(c0 + j) * size) : S;
                g[j] = in ? *reinterpret_cast<const float4*>(gain + (size_t)(c0 + j) * step) : S;
            }
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (c0 + j < count) {
                    *reinterpret_cast<float4*>(base + (size_t)(c0 + j) * size) = S;
                    S.x = fmaf(g[j].x, S.x, add[j].x);
                    S.y = fmaf(g[j].y, S.y, add[j].y);
                    S.z = fmaf(g[j].z, S.z, add[j].z);
                    S.w = fmaf(g[j].w, S.w, add[j].w);
                }
        }
    } else {
        // eight chunks' loads are under way all the time (they do not depend on the carried value): a slot takes the next one as soon as it is used
        float4 add[8];
        float g[8];
        auto load = [&](int j, int c) {
            const bool in = c < count;
            add[j] = in ? *reinterpret_cast<const float4*>(base + (size_t)c * size) : S;
            g[j] = in ? gain[(size_t)c * step] : 1.0f;
        };
#pragma unroll
        for (int j = 0; j < 8; ++j) load(j, j);
        for (int c0 = 0; c0 < count; c0 += 8) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (c0 + j < count) {
                    const float4 x = add[j];
                    const float f = g[j];
                    load(j, c0 + 8 + j);
                    *reinterpret_cast<float4*>(base + (size_t)(c0 + j) * size) = S;
                    S = make_float4(fmaf(f, S.x, x.x), fmaf(f, S.y, x.y), fmaf(f, S.z, x.z), fmaf(f, S.w, x.w));
                }
        }
    }
    st[0] = S.x;
    st[1] = S.y;
    st[2] = S.z;
    st[3] = S.w;
}

// ---- the outputs of a chunk: diag(gamma) Q S + (Q K^T, decayed and masked) U --------------------------------------------------
// Two blocks per SM (104 KB each): the planes of q (then of the scores) and of one other operand: S's first 64 rows (of dv), its others, k, u.
// A warp has 32 tokens and sixteen columns of each half of dv.  Bound by the tensor cores (mma.sync: 8.2 cycles for 16 x 8 x 16 per
// quarter of an SM, 59 us of 153 for 3,000 tokens, 32 heads of 128 x 128); with fragments split by every warp that needs them 164 us.
template <int DK, int DV>
__global__ void __launch_bounds__(256, 2) lc_output_kernel(LcArgs a, const float* __restrict__ values, size_t ldu) {
    extern __shared__ __align__(16) float lc_smem[];
    constexpr int WIDE = DK > DV ? DK : DV, PK = lc_plane<DK>(64), PV = lc_plane<DV>(64), PS = lc_plane<64>(64), HALVES = DV / 64;
    const uint32_t pq = (uint32_t)__cvta_generic_to_shared(lc_smem), px = pq + 3 * PK;
    float* fx = lc_smem + LC_C * LC_LP;          // (a chunk that holds a NaN or an infinity: the scores and u as they are)
    static_assert(3 * PK + 3 * lc_plane<WIDE>(64) >= (LC_C * LC_LP + LC_C * LC_LD) * 4, "they fit");
    __shared__ double sb[LC_C];
    const int h = blockIdx.x, c = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t0 = a.chunk_meta[4 * c], cnt = a.chunk_meta[4 * c + 1];
    const int kh = h / (a.H / a.G);
    const float* S = a.states + ((size_t)c * a.H + h) * a.dv * a.dk;
    {
        LcTile<DK> tq, ts;
        tq.load(a.q + (size_t)t0 * a.ldq + (size_t)kh * a.dk, a.ldq, cnt, a.dk);
        ts.load(S, a.dk, min(64, a.dv), a.dk);
        lc_decays(a.gate, a.head_decay, t0, cnt, a.H, h, sb);
        tq.to_planes(pq);
        ts.to_planes(px);
    }
    const int m0 = (warp & 1) * 32, wn = warp >> 1, t = lane & 3, g = lane >> 2;
    float acc[HALVES][2][2][4];                  // [half of dv][16 rows][8 columns]
    lc_zero<HALVES * 16>(&acc[0][0][0][0]);
    __syncthreads();
#pragma unroll
    for (int b = 0; b < HALVES; ++b) {
        float low[2][2][4];
        lc_zero<16>(&low[0][0][0]);
#pragma unroll 2
        for (int k0 = 0; k0 < DK; k0 += 16) {
            LcA fa[2];
            LcB fb[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) fa[i] = lc_a_mk<DK + 8>(pq + ((m0 + 16 * i) * (DK + 8) + k0) * 2, PK);
            lc_b2_nk<DK + 8>(px + (wn * 16 * (DK + 8) + k0) * 2, PK, fb);
            lc_products<2, 2>(acc[b], low, fa, fb);
        }
        lc_add<16>(&acc[b][0][0][0], &low[0][0][0]);
        __syncthreads();
        LcTile<DK> next;
        if (b + 1 < HALVES) next.load(a.dv > 64 ? S + (size_t)64 * a.dk : S, a.dk, a.dv - 64, a.dk);
        else next.load(a.k + (size_t)t0 * a.ldk + (size_t)kh * a.dk, a.ldk, cnt, a.dk);
        next.to_planes(px);
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const float g0 = lc_exp(sb[m0 + 16 * i + g]), g1 = lc_exp(sb[m0 + 16 * i + g + 8]);
#pragma unroll
        for (int b = 0; b < HALVES; ++b)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                acc[b][i][j][0] *= g0;
                acc[b][i][j][1] *= g0;
                acc[b][i][j][2] *= g1;
                acc[b][i][j][3] *= g1;
            }
    }
    // scores of the rows m0.. and keys 16 wn..: nothing to do above the diagonal
    float sc[2][2][4];                           // [16 rows][8 columns]
    {
        float low[2][2][4];
        lc_zero<16>(&sc[0][0][0]);
        lc_zero<16>(&low[0][0][0]);
        if (wn * 16 <= m0 + 31) {
#pragma unroll 2
            for (int k0 = 0; k0 < DK; k0 += 16) {
                LcA fa[2];
                LcB fb[2];
#pragma unroll
                for (int i = 0; i < 2; ++i) fa[i] = lc_a_mk<DK + 8>(pq + ((m0 + 16 * i) * (DK + 8) + k0) * 2, PK);
                lc_b2_nk<DK + 8>(px + (wn * 16 * (DK + 8) + k0) * 2, PK, fb);
                lc_products<2, 2>(sc, low, fa, fb);
            }
            lc_add<16>(&sc[0][0][0], &low[0][0][0]);
        }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const int m = m0 + 16 * i + g + 8 * (x >> 1), n = wn * 16 + 8 * j + 2 * t + (x & 1);
                sc[i][j][x] = n <= m ? sc[i][j][x] * lc_exp(sb[m] - sb[n]) : 0.0f;
            }
    LcTile<DV> tu;
    tu.load(values + (size_t)t0 * ldu + (size_t)h * a.dv, ldu, cnt, a.dv);
    const bool plain = !__syncthreads_or(tu.not_finite());      // ... and every warp is through with q and k
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int m = m0 + 16 * i + g + 8 * half, n = wn * 16 + 8 * j + 2 * t;
                if (plain) {
                    const LcSplit p = lc_split(sc[i][j][2 * half], sc[i][j][2 * half + 1]);
                    const uint32_t to = pq + (m * 72 + n) * 2;
                    lc_sts32(to, p.h);
                    lc_sts32(to + PS, p.m);
                    lc_sts32(to + 2 * PS, p.l);
                } else {
                    *reinterpret_cast<float2*>(lc_smem + m * LC_LP + n) = make_float2(sc[i][j][2 * half], sc[i][j][2 * half + 1]);
                }
            }
    if (plain) tu.to_planes(px);
    else tu.to_floats(fx);
    __syncthreads();
#pragma unroll
    for (int b = 0; b < HALVES; ++b) {
        if (!plain) {
            lc_causal(acc[b], lc_smem, fx + 64 * b, m0, wn);
            continue;
        }
        float low[2][2][4];
        lc_zero<16>(&low[0][0][0]);
        for (int k0 = 0; k0 < m0 + 32; k0 += 16) {
            LcA fa[2];
            LcB fb[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) fa[i] = lc_a_mk<72>(pq + ((m0 + 16 * i) * 72 + k0) * 2, PS);
            lc_b2_kn<DV + 8>(px + (k0 * (DV + 8) + 64 * b + wn * 16) * 2, PV, fb);
            lc_products<2, 2>(acc[b], low, fa, fb);
        }
        lc_add<16>(&acc[b][0][0][0], &low[0][0][0]);
    }
#pragma unroll
    for (int b = 0; b < HALVES; ++b)
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int n = 64 * b + wn * 16 + 8 * j + 2 * t;
                if (n >= a.dv) continue;
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const int m = m0 + 16 * i + g + 8 * half;
                    if (m < cnt)
                        *reinterpret_cast<float2*>(a.out + ((size_t)(t0 + m) * a.H + h) * a.dv + n) =
                            make_float2(acc[b][i][j][2 * half], acc[b][i][j][2 * half + 1]);
                }
            }
}

// ---- the delta rule ---------------------------------------------------------------------------------------------------------
// T = (I + L)^-1 by blocks: the four 16 x 16 blocks on the diagonal by substitution, a column per thread; then twice the inverse of a
// matrix of two by two blocks, [A 0; B D]^-1 = [A^-1 0; -D^-1 B A^-1, D^-1].  The part of T above its diagonal blocks is scratch.
__device__ __forceinline__ void lc_invert(const float* __restrict__ L, float* __restrict__ T) {
    const int tid = threadIdx.x;
    if (tid < 64) {
        const int b = (tid >> 4) * 16, j = tid & 15;
        float x[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            float s = i == j ? 1.0f : 0.0f;
#pragma unroll
            for (int p = 0; p < i; ++p) s = fmaf(-L[(b + i) * LC_LP + b + p], x[p], s);
            x[i] = s;
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) T[(b + i) * LC_LP + b + j] = x[i];
    }
    __syncthreads();
    // pairs of 16: blocks (1, 0) and (3, 2); the product in between goes to blocks (0, 1) and (2, 3)
    const int b16 = (tid >> 7) * 32, r16 = (tid & 127) >> 3, c16 = (tid & 7) * 2;
    {
        float s0 = 0.0f, s1 = 0.0f;
#pragma unroll
        for (int p = 0; p < 16; ++p) {
            const float x = L[(b16 + 16 + r16) * LC_LP + b16 + p];
            s0 = fmaf(x, T[(b16 + p) * LC_LP + b16 + c16], s0);
            s1 = fmaf(x, T[(b16 + p) * LC_LP + b16 + c16 + 1], s1);
        }
        T[(b16 + r16) * LC_LP + b16 + 16 + c16] = s0;
        T[(b16 + r16) * LC_LP + b16 + 16 + c16 + 1] = s1;
    }
    __syncthreads();
    {
        float s0 = 0.0f, s1 = 0.0f;
#pragma unroll
        for (int p = 0; p < 16; ++p) {
            const float x = T[(b16 + 16 + r16) * LC_LP + b16 + 16 + p];
            s0 = fmaf(-x, T[(b16 + p) * LC_LP + b16 + 16 + c16], s0);
            s1 = fmaf(-x, T[(b16 + p) * LC_LP + b16 + 16 + c16 + 1], s1);
        }
        T[(b16 + 16 + r16) * LC_LP + b16 + c16] = s0;
        T[(b16 + 16 + r16) * LC_LP + b16 + c16 + 1] = s1;
    }
    __syncthreads();
    // the pair of 32: T[32.., 0..] = -T[32.., 32..] L[32.., 0..] T[0.., 0..]; both triangles' upper blocks are scratch by now and count as zero
    const int r = tid >> 3, c = (tid & 7) * 4;
    {
        float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        const int from = c & 16;                 // T[0..32, 0..32] is zero above its diagonal blocks
        for (int p = from; p < 32; ++p) {
            const float x = L[(32 + r) * LC_LP + p];
            const float4 y = *reinterpret_cast<const float4*>(T + p * LC_LP + c);
            s[0] = fmaf(x, y.x, s[0]);
            s[1] = fmaf(x, y.y, s[1]);
            s[2] = fmaf(x, y.z, s[2]);
            s[3] = fmaf(x, y.w, s[3]);
        }
        *reinterpret_cast<float4*>(T + r * LC_LP + 32 + c) = make_float4(s[0], s[1], s[2], s[3]);
    }
    __syncthreads();
    {
        float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        const int to = (r & 16) + 16;
        for (int p = 0; p < to; ++p) {
            const float x = T[(32 + r) * LC_LP + 32 + p];
            const float4 y = *reinterpret_cast<const float4*>(T + p * LC_LP + 32 + c);
            s[0] = fmaf(-x, y.x, s[0]);
            s[1] = fmaf(-x, y.y, s[1]);
            s[2] = fmaf(-x, y.z, s[2]);
            s[3] = fmaf(-x, y.w, s[3]);
        }
        *reinterpret_cast<float4*>(T + (32 + r) * LC_LP + c) = make_float4(s[0], s[1], s[2], s[3]);
    }
    __syncthreads();
}

// W = T diag(beta gamma) K, U0 = T diag(beta) V of a chunk, and what else the chain needs: its gain, and W and K' = diag(gamma_C / gamma) K as the
// fragments that the chain's warps multiply, split and in the order of their lanes: a 16-byte word per lane and part, for W by rows of
// 16 tokens and steps of sixteen channels, for K' by eight channels and 32 tokens.  (A product's result has the places of the next one's
// first operand, so W goes out as it comes.)  Bound by the tensor cores.
template <int DK>
struct LcFrag {
    static constexpr int W = 4 * (DK / 16) * 3 * 32, K = (DK / 8) * 2 * 3 * 32, SIZE = W + K;      // words
};
__device__ __forceinline__ void lc_put_frag(uint4* to, const LcSplit& x, const LcSplit& y, const LcSplit& z, const LcSplit& w) {
    const int lane = threadIdx.x & 31;
    to[lane] = make_uint4(x.h, y.h, z.h, w.h);
    to[32 + lane] = make_uint4(x.m, y.m, z.m, w.m);
    to[64 + lane] = make_uint4(x.l, y.l, z.l, w.l);
}
template <int DK, int DV>
__global__ void __launch_bounds__(256, 2) lc_delta_prepare_kernel(LcArgs a) {
    extern __shared__ __align__(16) float lc_smem[];
    float* sk = lc_smem;                         // [64][LC_LD]
    float* sv = sk + LC_C * LC_LD;               // [64][LC_LD]
    float* sL = sv + LC_C * LC_LD;               // [64][LC_LP]
    float* sT = sL + LC_C * LC_LP;               // [64][LC_LP]
    __shared__ double sb[LC_C];
    __shared__ float sbeta[LC_C], sbg[LC_C], sr[LC_C];
    const int h = blockIdx.x, c = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t0 = a.chunk_meta[4 * c], cnt = a.chunk_meta[4 * c + 1];
    const int kh = h / (a.H / a.G);
    lc_load<DK, LC_LD>(sk, a.k + (size_t)t0 * a.ldk + (size_t)kh * a.dk, a.ldk, cnt, a.dk);
    lc_commit();
    lc_load<DV, LC_LD>(sv, a.v + (size_t)t0 * a.ldv + (size_t)h * a.dv, a.ldv, cnt, a.dv);
    lc_commit();
    lc_decays(a.gate, a.head_decay, t0, cnt, a.H, h, sb);
    bool odd = false;                            // a NaN or an infinity
    if (threadIdx.x < LC_C) {
        const int t = threadIdx.x;
        const float b = t < cnt ? a.beta[(size_t)(t0 + t) * a.H + h] : 0.0f;
        odd = !(fabsf(b) < INFINITY && fabs(sb[t]) < INFINITY);
        sbeta[t] = b;
        sbg[t] = b * lc_exp(sb[t]);
        sr[t] = lc_exp(sb[LC_C - 1] - sb[t]);
        if (t == 0) a.gain[(size_t)c * a.H + h] = lc_exp(sb[LC_C - 1]);
    }
    const int m0 = (warp & 1) * 32, wn = warp >> 1, t = lane & 3, g = lane >> 2;
    uint4* fw = a.frag + ((size_t)c * a.H + h) * LcFrag<DK>::SIZE;
    uint4* fk = fw + LcFrag<DK>::W;
    lc_wait<1>();
    __syncthreads();
    for (int item = warp; item < DK / 8 * 2; item += 8) {       // K': eight channels and 32 tokens
        LcSplit x[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int row = (item & 1) * 32 + 8 * e + 2 * t;
            const float* p = sk + row * LC_LD + (item >> 1) * 8 + g;
            x[e] = lc_split(p[0], sr[row], p[LC_LD], sr[row + 1]);
        }
        lc_put_frag(fk + item * 96, x[0], x[1], x[2], x[3]);
    }
    {
        float s[2][2][4], s_low[2][2][4];        // [8 columns][16 rows]
        lc_zero<16>(&s[0][0][0]);
        lc_zero<16>(&s_low[0][0][0]);
        if (wn * 16 <= m0 + 31) {
#pragma unroll 1
            for (int k0 = 0; k0 < DK; k0 += 16) {
                LcA fa[2];
#pragma unroll
                for (int i = 0; i < 2; ++i) fa[i] = lc_a_rows(sk + (m0 + 16 * i) * LC_LD + k0, LC_LD);
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const LcB fb = lc_b_rows(sk + (wn * 16 + 8 * j) * LC_LD + k0, LC_LD);
                    lc_one(s[j], s_low[j], fa, fb);
                }
            }
            lc_add<16>(&s[0][0][0], &s_low[0][0][0]);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    const int m = m0 + 16 * i + g + 8 * (x >> 1), n = wn * 16 + 8 * j + 2 * t + (x & 1);
                    sL[m * LC_LP + n] = n < m ? s[j][i][x] * sbeta[m] * lc_exp(sb[m] - sb[n]) : 0.0f;
                }
    }
    lc_wait<0>();
    odd |= lc_not_finite<DK, LC_LD>(sk) || lc_not_finite<DV, LC_LD>(sv);
    if (__syncthreads_or(odd)) {                 // W and U0 by substitution, a column per thread, in place: no row takes part in one before it
        if (threadIdx.x < DK + DV) {
            const bool key = threadIdx.x < DK;
            float* col = key ? sk + threadIdx.x : sv + (threadIdx.x - DK);
            for (int m = 0; m < LC_C; ++m) {
                float x = (key ? sbg : sbeta)[m] * col[m * LC_LD];
                for (int p = 0; p < m; ++p) x = fmaf(-sL[m * LC_LP + p], col[p * LC_LD], x);
                col[m * LC_LD] = x;
            }
        }
        __syncthreads();
        for (int item = warp; item < 4 * (DK / 16); item += 8) {
            const float* p = sk + (item / (DK / 16) * 16 + g) * LC_LD + item % (DK / 16) * 16 + 2 * t;
            lc_put_frag(fw + item * 96, lc_split(p[0], p[1]), lc_split(p[8 * LC_LD], p[8 * LC_LD + 1]), lc_split(p[8], p[9]),
                        lc_split(p[8 * LC_LD + 8], p[8 * LC_LD + 9]));
        }
        for (int idx = threadIdx.x; idx < cnt * a.dv; idx += 256) a.u[((size_t)(t0 + idx / a.dv) * a.H + h) * a.dv + idx % a.dv] = sv[idx / a.dv * LC_LD + idx % a.dv];
        return;
    }
    lc_invert(sL, sT);
    // both products: rows m0 + 16 i (32 per warp pair), columns wn * (COLS / 4)..; T has nothing to the right of its diagonal blocks
    auto product = [&](const float* s, const float* scale, int cols, int width, float* o, size_t ld, auto tiles, auto as_fragments) {
        constexpr int NT = decltype(tiles)::value;
        float acc[NT][2][4], low[NT][2][4];      // [8 columns][16 rows]
        lc_zero<NT * 8>(&acc[0][0][0]);
        lc_zero<NT * 8>(&low[0][0][0]);
        for (int k0 = 0; k0 < m0 + 32; k0 += 16) {
            const LcScale f = lc_scale(scale + k0);
            LcA fa[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const bool right = k0 >= m0 + 16 * i + 16;       // scratch: counts as zero
                fa[i] = right ? LcA{} : lc_a_rows4(sT + (m0 + 16 * i) * LC_LP + k0, LC_LP, f);
            }
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                const LcB fb = lc_b_cols(s + k0 * LC_LD + wn * width + 8 * j, LC_LD);
                lc_one(acc[j], low[j], fa, fb);
            }
        }
        lc_add<NT * 8>(&acc[0][0][0], &low[0][0][0]);
        if constexpr (decltype(as_fragments)::value) {
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < NT; j += 2)
                    lc_put_frag(fw + ((m0 / 16 + i) * (DK / 16) + (wn * width + 8 * j) / 16) * 96, lc_split(acc[j][i][0], acc[j][i][1]), lc_split(acc[j][i][2], acc[j][i][3]),
                                lc_split(acc[j + 1][i][0], acc[j + 1][i][1]), lc_split(acc[j + 1][i][2], acc[j + 1][i][3]));
            return;
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                const int n = wn * width + 8 * j + 2 * t;
                if (n >= cols) continue;
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const int m = m0 + 16 * i + g + 8 * half;
                    if (m < cnt) *reinterpret_cast<float2*>(o + (size_t)m * ld + n) = make_float2(acc[j][i][2 * half], acc[j][i][2 * half + 1]);
                }
            }
    };
    product(sk, sbg, a.dk, DK / 4, nullptr, 0, std::integral_constant<int, DK / 32>{}, std::true_type{});
    product(sv, sbeta, a.dv, DV / 4, a.u + ((size_t)t0 * a.H + h) * a.dv, (size_t)a.H * a.dv, std::integral_constant<int, DV / 32>{}, std::false_type{});
}

// U = U0 - W S and S' = gamma_C S + K'^T U, chunk after chunk, for 16 NG columns of one head's S per block: a chain of two products per chunk.
// W and K' come as fragments straight into the registers of the warps that multiply them, the next chunk's while the current one is worked on;
// S and U are split by the threads that make them and pass through shared memory as planes.  In the first product warp w has rows 16 (w % 4)
// of U and a quarter of the key channels; the quarters meet in a pass over U.  In the second warp w has eight key channels of
// S^T = U^T K' and all columns: S stays in its registers.
// Bound by the tensor cores (24 products of 16 x 8 x 16 per warp and half of a chunk), what they read from shared memory, three barriers, and
// the fragments' way from L2 (96 KB per block and chunk): 64 chunks take 179 us.  Warps that split all that they multiply took 238; with W
// and K' split by eight more warps into planes in shared memory 206, bound by the reads and writes there.
#define LC_CARRY_THREADS 512
template <int DK, int NG>
struct LcCarryShared {
    static constexpr int NS = 16 * NG, PS = lc_plane<DK>(NS), PU = lc_plane<NS>(64), LQ = NS + 4;
    // bytes: the planes of S^T [NS][dk] and U [64][NS], the quarters of W S
    static constexpr int S = 0, U = S + 3 * PS, SUM = U + 3 * PU, SIZE = SUM + 4 * LC_C * LQ * 4;
};
template <int DK, int NG>
__global__ void __launch_bounds__(LC_CARRY_THREADS, 1) lc_delta_carry_kernel(LcArgs a) {
    using M = LcCarryShared<DK, NG>;
    constexpr int NS = M::NS;
    extern __shared__ __align__(16) float lc_smem[];
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(lc_smem);
    const int h = blockIdx.y, r = blockIdx.z, n_base = blockIdx.x * NS, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int first = a.req_chunks[2 * r], count = a.req_chunks[2 * r + 1];
    if (count <= 0) return;
    const int t = lane & 3, g = lane >> 2;
    // fragments: the warp's steps of W, its channels of K'
    constexpr int STEPS = DK / 64;
    const bool has = warp * 8 < DK;
    uint4 fw[STEPS][3], fk[2][3];
    auto load_w = [&](int c) {
        const uint4* p = a.frag + ((size_t)c * a.H + h) * LcFrag<DK>::SIZE + ((warp & 3) * (DK / 16) + (warp >> 2) * STEPS) * 96 + lane;
#pragma unroll
        for (int e = 0; e < STEPS; ++e)
#pragma unroll
            for (int part = 0; part < 3; ++part) fw[e][part] = __ldg(p + (e * 3 + part) * 32);
    };
    auto load_k = [&](int c) {
        const uint4* p = a.frag + ((size_t)c * a.H + h) * LcFrag<DK>::SIZE + LcFrag<DK>::W + warp * 192 + lane;
        if (has)
#pragma unroll
            for (int e = 0; e < 2; ++e)
#pragma unroll
                for (int part = 0; part < 3; ++part) fk[e][part] = __ldg(p + (e * 3 + part) * 32);
    };
    // S^T of key channels 8 warp.. (if there are so many): of every sixteen columns rows g and g + 8, channels 2t and 2t + 1
    const int m = warp * 8 + 2 * t;
    float S[NG][4];
    float* st = a.state + (size_t)a.slots[r] * a.state_stride + (size_t)h * a.dv * a.dk;
    {
        const bool fresh = a.positions[a.chunk_meta[4 * first]] == 0;
#pragma unroll
        for (int b = 0; b < NG; ++b)
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const int n = n_base + 16 * b + g + 8 * (x >> 1);
                S[b][x] = (!fresh && has && m + (x & 1) < a.dk && n < a.dv) ? st[(size_t)n * a.dk + m + (x & 1)] : 0.0f;
            }
    }
    auto to_planes = [&]() {
        if (!has) return;
#pragma unroll
        for (int b = 0; b < NG; ++b)
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const LcSplit x = lc_split(S[b][2 * half], S[b][2 * half + 1]);
                const uint32_t to = base + M::S + ((16 * b + g + 8 * half) * (DK + 8) + m) * 2;
                lc_sts32(to, x.h);
                lc_sts32(to + M::PS, x.m);
                lc_sts32(to + 2 * M::PS, x.l);
            }
    };
    // the pass over U: a thread's row and two of every sixteen columns
    const int row = threadIdx.x >> 3, col = (threadIdx.x & 7) * 2;
    float* sum = lc_smem + M::SUM / 4;
    auto u_place = [&](int t0, int b) { return a.u + ((size_t)(t0 + row) * a.H + h) * a.dv + n_base + 16 * b + col; };
    load_w(first);
    load_k(first);
    to_planes();
    int t0 = a.chunk_meta[4 * first], cnt = a.chunk_meta[4 * first + 1];
    for (int i = 0; i < count; ++i) {
        const int c = first + i;
        const float gain = __ldg(a.gain + (size_t)c * a.H + h);
        float2 u[NG];
#pragma unroll
        for (int b = 0; b < NG; ++b)
            u[b] = row < cnt && n_base + 16 * b + col < a.dv ? *reinterpret_cast<const float2*>(u_place(t0, b)) : make_float2(0.0f, 0.0f);
        int next_t0 = 0, next_cnt = 0;
        if (i + 1 < count) {
            next_t0 = a.chunk_meta[4 * (c + 1)];
            next_cnt = a.chunk_meta[4 * (c + 1) + 1];
        }
        __syncthreads();                         // S's planes
        {
            const int m0 = (warp & 3) * 16, part = warp >> 2;
            float p[1][2 * NG][4], low[1][2 * NG][4];
            lc_zero<8 * NG>(&p[0][0][0]);
            lc_zero<8 * NG>(&low[0][0][0]);
#pragma unroll
            for (int e = 0; e < STEPS; ++e) {
                const int k0 = (part * STEPS + e) * 16;
                const LcA fa = {{{fw[e][0].x, fw[e][1].x, fw[e][2].x}, {fw[e][0].y, fw[e][1].y, fw[e][2].y}, {fw[e][0].z, fw[e][1].z, fw[e][2].z},
                                 {fw[e][0].w, fw[e][1].w, fw[e][2].w}}};
                LcB fb[2 * NG];
#pragma unroll
                for (int b = 0; b < NG; ++b) lc_b2_nk<DK + 8>(base + M::S + (16 * b * (DK + 8) + k0) * 2, M::PS, fb + 2 * b);
                lc_products<1, 2 * NG>(p, low, &fa, fb);
            }
            if (i + 1 < count) load_w(c + 1);
            lc_add<8 * NG>(&p[0][0][0], &low[0][0][0]);
#pragma unroll
            for (int j = 0; j < 2 * NG; ++j)
#pragma unroll
                for (int half = 0; half < 2; ++half)
                    *reinterpret_cast<float2*>(sum + (part * LC_C + m0 + g + 8 * half) * M::LQ + 8 * j + 2 * t) = make_float2(p[0][j][2 * half], p[0][j][2 * half + 1]);
        }
        {   // what the chunk starts from, as [dv, dk]
            float* o = a.states + ((size_t)c * a.H + h) * a.dv * a.dk;
#pragma unroll
            for (int b = 0; b < NG; ++b)
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const int n = n_base + 16 * b + g + 8 * half;
                    if (has && m < a.dk && n < a.dv) *reinterpret_cast<float2*>(o + (size_t)n * a.dk + m) = make_float2(S[b][2 * half], S[b][2 * half + 1]);
                }
        }
        __syncthreads();                         // the quarters
#pragma unroll
        for (int b = 0; b < NG; ++b) {
            float2 x[4];
#pragma unroll
            for (int part = 0; part < 4; ++part) x[part] = *reinterpret_cast<const float2*>(sum + (part * LC_C + row) * M::LQ + 16 * b + col);
            u[b].x -= (x[0].x + x[1].x) + (x[2].x + x[3].x);
            u[b].y -= (x[0].y + x[1].y) + (x[2].y + x[3].y);
            if (row < cnt && n_base + 16 * b + col < a.dv) *reinterpret_cast<float2*>(u_place(t0, b)) = u[b];
            const LcSplit y = lc_split(u[b].x, u[b].y);
            const uint32_t to = base + M::U + (row * (NS + 8) + 16 * b + col) * 2;
            lc_sts32(to, y.h);
            lc_sts32(to + M::PU, y.m);
            lc_sts32(to + 2 * M::PU, y.l);
        }
        __syncthreads();                         // U's planes
        if (has) {
            float p[NG][1][4], low[NG][1][4];
            lc_zero<4 * NG>(&p[0][0][0]);
            lc_zero<4 * NG>(&low[0][0][0]);
#pragma unroll
            for (int step = 0; step < 4; ++step) {
                LcA fa[NG];
#pragma unroll
                for (int b = 0; b < NG; ++b) fa[b] = lc_a_km<NS + 8>(base + M::U + (16 * step * (NS + 8) + 16 * b) * 2, M::PU);
                const uint4* f = fk[step >> 1];
                const LcB fb = step & 1 ? LcB{{{f[0].z, f[1].z, f[2].z}, {f[0].w, f[1].w, f[2].w}}} : LcB{{{f[0].x, f[1].x, f[2].x}, {f[0].y, f[1].y, f[2].y}}};
                lc_products<NG, 1>(p, low, fa, &fb);
            }
            if (i + 1 < count) load_k(c + 1);
            lc_add<4 * NG>(&p[0][0][0], &low[0][0][0]);
#pragma unroll
            for (int b = 0; b < NG; ++b)
#pragma unroll
                for (int x = 0; x < 4; ++x) S[b][x] = fmaf(gain, S[b][x], p[b][0][x]);
        }
        to_planes();                             // (read by all before the second barrier)
        t0 = next_t0;
        cnt = next_cnt;
    }
#pragma unroll
    for (int b = 0; b < NG; ++b)
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            const int n = n_base + 16 * b + g + 8 * (x >> 1);
            if (has && m + (x & 1) < a.dk && n < a.dv) st[(size_t)n * a.dk + m + (x & 1)] = S[b][x];
        }
}

// ---- a forget gate per key channel (csrc/linear_state.cu): k_t = 1 - f_t, S_t = diag(f_t) S_(t-1) + k_t v_t^T -------------------------
// The ratio of two tokens' decays is a product of gates per channel, so it rides on q and k.  A chunk is cut into four runs of
// 16 tokens, and every product of gates is made forward or backward inside a run (F: over a whole run), so none is a quotient and
// none exceeds 1:
//   q'_t = q_t prod(u <= t in t's run) f_u,     k'_s = k_s prod(u > s in s's run) f_u;
//   scores between runs i > j: q'_t diag(prod of F between j and i) k'_s;    from the state: q'_t diag(prod of F before i) S;
//   to the state: k'_s diag(prod of F behind j);    inside a run, where the product would have to be taken apart, token by token.
#define LC_RUN 16

template <int DK, int DV>
__global__ void __launch_bounds__(256, 2) lc_forget_state_kernel(LcArgs a) {
    extern __shared__ __align__(16) float lc_smem[];
    float* sf = lc_smem;                         // [64][LC_LD]: f, then what k becomes
    float* sv = sf + LC_C * LC_LD;               // [64][LC_LD]
    __shared__ float sF[4][DK], sr[LC_C];
    const int h = blockIdx.x, c = blockIdx.y;
    const int t0 = a.chunk_meta[4 * c], cnt = a.chunk_meta[4 * c + 1];
    lc_load<DK, LC_LD>(sf, a.k + (size_t)t0 * a.ldk + (size_t)h * a.dk, a.ldk, cnt, a.dk);
    lc_load<DV, LC_LD>(sv, a.v + (size_t)t0 * a.ldv + (size_t)h * a.dv, a.ldv, cnt, a.dv);
    lc_commit();
    if (threadIdx.x < LC_C) sr[threadIdx.x] = 1.0f;
    lc_wait<0>();
    __syncthreads();
    constexpr int PER = DK / 64;                 // runs per thread; a thread owns one channel
    const int ch = threadIdx.x % DK, first = threadIdx.x / DK * PER;
    float kk[PER][LC_RUN];
#pragma unroll
    for (int u = 0; u < PER; ++u) {
        float r = 1.0f;
#pragma unroll
        for (int s = LC_RUN - 1; s >= 0; --s) {
            const int t = (first + u) * LC_RUN + s;
            const bool in = t < cnt && ch < a.dk;
            const float f = in ? sf[t * LC_LD + ch] : 1.0f;
            kk[u][s] = in ? (1.0f - f) * r : 0.0f;
            r *= f;
        }
        sF[first + u][ch] = r;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < PER; ++u) {
        float behind = 1.0f;
        for (int m = first + u + 1; m < 4; ++m) behind *= sF[m][ch];
#pragma unroll
        for (int s = 0; s < LC_RUN; ++s) sf[((first + u) * LC_RUN + s) * LC_LD + ch] = kk[u][s] * behind;
    }
    if (first == 0 && ch < a.dk) a.gain[((size_t)c * a.H + h) * a.dk + ch] = sF[0][ch] * sF[1][ch] * sF[2][ch] * sF[3][ch];
    __syncthreads();
    lc_add_up<DK, DV, true>(a, h, c, sf, sv, sr);
}

// Two blocks per SM: q (then q', then the scores), f (then k'), and a buffer for S's halves and then v.
template <int DK, int DV>
__global__ void __launch_bounds__(256, 2) lc_forget_output_kernel(LcArgs a) {
    extern __shared__ __align__(16) float lc_smem[];
    float* sq = lc_smem;
    float* sf = sq + LC_C * LC_LD;
    float* sx = sf + LC_C * LC_LD;
    __shared__ __align__(16) float sF[4][DK], sbefore[4][DK], sone[DK], smid[DK];      // a run's product; of the runs before one; 1; of runs 1 and 2
    const int h = blockIdx.x, c = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t0 = a.chunk_meta[4 * c], cnt = a.chunk_meta[4 * c + 1];
    const float* S = a.states + ((size_t)c * a.H + h) * a.dv * a.dk;
    lc_load<DK, LC_LD>(sq, a.q + (size_t)t0 * a.ldq + (size_t)h * a.dk, a.ldq, cnt, a.dk);
    lc_load<DK, LC_LD>(sf, a.k + (size_t)t0 * a.ldk + (size_t)h * a.dk, a.ldk, cnt, a.dk);
    lc_commit();
    lc_load<DK, LC_LD>(sx, S, a.dk, min(64, a.dv), a.dk);
    lc_commit();
    lc_wait<1>();
    __syncthreads();
    // inside the runs: thread (run, s, channels 4 cl.. of every 16) carries k_s through the tokens t >= s
    const int run = threadIdx.x >> 6, ds = (threadIdx.x & 63) >> 2, cl = threadIdx.x & 3;
    float inner[LC_RUN];
#pragma unroll
    for (int t = 0; t < LC_RUN; ++t) inner[t] = 0.0f;
#pragma unroll 1
    for (int e = 0; e < DK; e += 16) {
        const float* fq = sq + run * LC_RUN * LC_LD + e + 4 * cl;
        const float* ff = sf + run * LC_RUN * LC_LD + e + 4 * cl;
        float4 r = *reinterpret_cast<const float4*>(ff + ds * LC_LD);
        r = make_float4(1.0f - r.x, 1.0f - r.y, 1.0f - r.z, 1.0f - r.w);
#pragma unroll
        for (int t = 0; t < LC_RUN; ++t) {
            const float4 qv = *reinterpret_cast<const float4*>(fq + t * LC_LD), fv = *reinterpret_cast<const float4*>(ff + t * LC_LD);
            if (t > ds) r = make_float4(r.x * fv.x, r.y * fv.y, r.z * fv.z, r.w * fv.w);
            if (t >= ds) inner[t] = fmaf(qv.x, r.x, fmaf(qv.y, r.y, fmaf(qv.z, r.z, fmaf(qv.w, r.w, inner[t]))));
        }
    }
#pragma unroll
    for (int t = 0; t < LC_RUN; ++t) {
        inner[t] += __shfl_xor_sync(0xffffffffu, inner[t], 1);
        inner[t] += __shfl_xor_sync(0xffffffffu, inner[t], 2);
    }
    __syncthreads();
    {   // q' and k' in place: a thread owns one channel of DK / 64 runs
        constexpr int PER = DK / 64;
        const int ch = threadIdx.x % DK, first = threadIdx.x / DK * PER;
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            float f[LC_RUN];
            float* pq = sq + (first + u) * LC_RUN * LC_LD + ch;
            float* pf = sf + (first + u) * LC_RUN * LC_LD + ch;
            float r = 1.0f;
#pragma unroll
            for (int s = 0; s < LC_RUN; ++s) {
                const bool in = (first + u) * LC_RUN + s < cnt && ch < a.dk;
                f[s] = in ? pf[s * LC_LD] : 1.0f;
                r *= f[s];
                pq[s * LC_LD] *= r;
            }
            sF[first + u][ch] = r;
            r = 1.0f;
#pragma unroll
            for (int s = LC_RUN - 1; s >= 0; --s) {
                pf[s * LC_LD] = (1.0f - f[s]) * r;
                r *= f[s];
            }
        }
    }
    __syncthreads();
    if (threadIdx.x < DK) {
        const int ch = threadIdx.x;
        sone[ch] = sbefore[0][ch] = 1.0f;
        float r = 1.0f;
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            r *= sF[m][ch];
            sbefore[m + 1][ch] = r;
        }
        smid[ch] = sF[1][ch] * sF[2][ch];
    }
    const int m0 = (warp & 1) * 32, wn = warp >> 1, t = lane & 3, g = lane >> 2;
    constexpr int HALVES = DV / 64;
    float acc[HALVES][2][2][4], low[HALVES][2][2][4];      // [half of dv][8 columns][16 rows]
    lc_zero<HALVES * 16>(&acc[0][0][0][0]);
    lc_zero<HALVES * 16>(&low[0][0][0][0]);
#pragma unroll
    for (int b = 0; b < HALVES; ++b) {
        lc_wait<0>();
        __syncthreads();
#pragma unroll 1
        for (int k0 = 0; k0 < DK; k0 += 16) {
            LcA fa[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) fa[i] = lc_a_rows_scaled(sq + (m0 + 16 * i) * LC_LD + k0, LC_LD, &sbefore[m0 / 16 + i][k0]);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const LcB fb = lc_b_rows(sx + (wn * 16 + 8 * j) * LC_LD + k0, LC_LD);
                lc_one(acc[b][j], low[b][j], fa, fb);
            }
        }
        __syncthreads();
        if (b + 1 < HALVES) lc_load<DK, LC_LD>(sx, a.dv > 64 ? S + (size_t)64 * a.dk : S, a.dk, a.dv - 64, a.dk);
        else lc_load<DV, LC_LD>(sx, a.v + (size_t)t0 * a.ldv + (size_t)h * a.dv, a.ldv, cnt, a.dv);
        lc_commit();
    }
    // between the runs: warp w < 6 takes one of the blocks (1,0) (2,0) (2,1) (3,0) (3,1) (3,2)
    float cross[1][2][4], cross_low[1][2][4];
    lc_zero<8>(&cross[0][0][0]);
    lc_zero<8>(&cross_low[0][0][0]);
    const int bi = warp == 0 ? 1 : warp < 3 ? 2 : 3, bj = warp == 0 ? 0 : warp < 3 ? warp - 1 : warp - 3;
    if (warp < 6) {
        const float* between = bi - bj == 1 ? sone : bi - bj == 2 ? sF[bi - 1] : smid;
#pragma unroll 2
        for (int k0 = 0; k0 < DK; k0 += 16) {
            const LcA fa = lc_a_rows_scaled(sq + bi * LC_RUN * LC_LD + k0, LC_LD, between + k0);
            const float* p = sf + bj * LC_RUN * LC_LD + k0;
            const LcB fb[2] = {lc_b_rows(p, LC_LD), lc_b_rows(p + 8 * LC_LD, LC_LD)};
            lc_products<1, 2>(cross, cross_low, &fa, fb);
        }
        lc_add<8>(&cross[0][0][0], &cross_low[0][0][0]);
    }
    __syncthreads();                             // every warp is through with q': the scores take its place
#pragma unroll
    for (int x = 0; x < LC_RUN; ++x)
        if ((x & 3) == cl) sq[(run * LC_RUN + x) * LC_LP + run * LC_RUN + ds] = x >= ds ? inner[x] : 0.0f;
    if (warp < 6) {
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int x = 0; x < 4; ++x) sq[(bi * LC_RUN + g + 8 * (x >> 1)) * LC_LP + bj * LC_RUN + 8 * j + 2 * t + (x & 1)] = cross[0][j][x];
    }
    lc_wait<0>();
    const bool plain = !__syncthreads_or(lc_not_finite<DV, LC_LD>(sx));
    if (!plain) {
#pragma unroll
        for (int b = 0; b < HALVES; ++b) lc_causal_cols(acc[b], sq, sx + 64 * b, m0, wn);
    }
    else for (int k0 = 0; k0 < m0 + 32; k0 += 16) {
        LcA fa[2];
#pragma unroll
        for (int i = 0; i < 2; ++i)              // nothing stands to the right of a row's own run
            fa[i] = k0 >= m0 + 16 * i + 16 ? LcA{} : lc_a_rows4(sq + (m0 + 16 * i) * LC_LP + k0, LC_LP);
#pragma unroll
        for (int b = 0; b < HALVES; ++b) {
            const float* p = sx + k0 * LC_LD + 64 * b + wn * 16;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const LcB fb = lc_b_cols(p + 8 * j, LC_LD);
                lc_one(acc[b][j], low[b][j], fa, fb);
            }
        }
    }
    lc_add<HALVES * 16>(&acc[0][0][0][0], &low[0][0][0][0]);
#pragma unroll
    for (int b = 0; b < HALVES; ++b)
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int n = 64 * b + wn * 16 + 8 * j + 2 * t;
                if (n >= a.dv) continue;
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const int m = m0 + 16 * i + g + 8 * half;
                    if (m < cnt)
                        *reinterpret_cast<float2*>(a.out + ((size_t)(t0 + m) * a.H + h) * a.dv + n) =
                            make_float2(acc[b][j][i][2 * half], acc[b][j][i][2 * half + 1]);
                }
            }
}

template <auto Kernel, typename... A>
static int lc_launch(dim3 grid, int threads, size_t smem, cudaStream_t s, A... args) {
    if (smem > 0 && !mm_allow_smem<Kernel>(smem)) {
        mm_set_last_error("linear state chunks: cannot reserve shared memory");
        return MM_ERR_LAUNCH;
    }
    mm_launch(Kernel, grid, dim3(threads), smem, s, args...);
    MM_CHECK_LAUNCH();
    return MM_OK;
}

template <int DK, int DV>
static int lc_run(const LcArgs& a, int n_requests, cudaStream_t s) {
    const dim3 chunks(a.H, a.n_chunks);
    const size_t tile = LC_C * LC_LD * sizeof(float), square = LC_C * LC_LP * sizeof(float);
    const size_t planes = 3 * lc_plane<DK>(64) + 3 * lc_plane<(DK > DV ? DK : DV)>(64);
    if (a.beta == nullptr) {
        if (const int rc = lc_launch<lc_state_kernel<DK, DV>>(chunks, 256, 2 * tile, s, a)) return rc;
        const long long size = (long long)a.H * a.dv * a.dk;
        if (const int rc = lc_launch<lc_carry_kernel<false>>(dim3(ceil_div(size / 4, 256), n_requests), 256, 0, s, a)) return rc;
        return lc_launch<lc_output_kernel<DK, DV>>(chunks, 256, planes, s, a, a.v, (size_t)a.ldv);
    }
    if (const int rc = lc_launch<lc_delta_prepare_kernel<DK, DV>>(chunks, 256, 2 * tile + 2 * square, s, a)) return rc;
    // Columns of S per block: sixteen, or 32 where that saves so many rounds of one block per SM that they make up for a chunk's time, which is 1.5 (dk 64)
    // to 1.6 times as long.  1,024 tokens, us with 16 and with 32 columns: 32 heads of 64 x 64, one portion (1 round and 1) 88 and 103, two (2, 1) 177 and
    // 162, four (4, 2) 342 and 308; 48 heads of 128 x 128 (3, 2) 291 and 304, 32 heads, two portions (4, 2) 376 and 345.
    const long long narrow = ceil_div((long long)ceil_div(a.dv, 16) * a.H * n_requests, 148), wide = ceil_div((long long)ceil_div(a.dv, 32) * a.H * n_requests, 148);
#define LC_CARRY(NG) lc_launch<lc_delta_carry_kernel<DK, NG>>(dim3(ceil_div(a.dv, 16 * NG), a.H, n_requests), LC_CARRY_THREADS, LcCarryShared<DK, NG>::SIZE, s, a)
    if (const int rc = 10 * narrow > 16 * wide ? LC_CARRY(2) : LC_CARRY(1)) return rc;
#undef LC_CARRY
    return lc_launch<lc_output_kernel<DK, DV>>(chunks, 256, planes, s, a, (const float*)a.u, (size_t)a.H * a.dv);
}

// 1 if the products take these sizes and pointers: heads of up to 128 numbers that are multiples of 4, rows and heads on 16-byte boundaries
MM_EXPORT int mm_linear_chunk_supported(const void* q, const void* k, const void* v, int ldq, int ldk, int ldv, const void* state,
                                        long long state_stride, int dk, int dv) {
    return dk > 0 && dv > 0 && dk <= 128 && dv <= 128 && dk % 4 == 0 && dv % 4 == 0 && ldq % 4 == 0 && ldk % 4 == 0 && ldv % 4 == 0 &&
           (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v) & 15) == 0 && state != nullptr && state_stride > 0;
}

// q, k, v, gate, beta (null: no delta rule), head_decay, out, state as for the walk (decays positive or zero); chunk_meta [chunks, 4] =
// (first token, tokens <= 64, request, .), req_chunks [requests, 2] = (first chunk, chunks).  Scratch, fp32: states [chunks, H, dv, dk], gain
// [chunks, H], and with beta frag [chunks, H, 12288] (24576 numbers for dk > 64), u [tokens, H, dv].
MM_EXPORT int mm_linear_chunk(const void* q, const void* k, const void* v, int ldq, int ldk, int ldv, const void* gate, const void* beta,
                              const void* head_decay, void* out, void* state, long long state_stride, const void* chunk_meta,
                              const void* req_chunks, const void* slots, const void* positions, int n_requests, int n_chunks, int H, int Gq,
                              int dk, int dv, void* states, void* gain, void* frag, void* u, void* stream) {
    MM_REQUIRE(H > 0 && Gq > 0 && H % Gq == 0, "linear state chunks: heads must be a positive multiple of the q/k heads");
    MM_REQUIRE(mm_linear_chunk_supported(q, k, v, ldq, ldk, ldv, state, state_stride, dk, dv), "linear state chunks: sizes or pointers that the products do not take");
    MM_REQUIRE(gate != nullptr || head_decay != nullptr, "linear state: a decay per token or per head is needed");
    MM_REQUIRE(out && slots && positions && chunk_meta && req_chunks && states && gain, "linear state chunks: the lists and the scratch are needed");
    MM_REQUIRE(beta == nullptr || (frag && u), "linear state chunks: the delta rule needs its scratch");
    MM_REQUIRE((((uintptr_t)out | (uintptr_t)states | (uintptr_t)frag | (uintptr_t)u) & 15) == 0, "linear state chunks: the scratch starts on 16-byte boundaries");
    MM_REQUIRE(n_chunks <= 65535 && n_requests <= 65535, "linear state chunks: too many chunks or requests");
    if (n_requests <= 0 || n_chunks <= 0) return MM_OK;
    LcArgs a;
    a.q = (const float*)q; a.k = (const float*)k; a.v = (const float*)v;
    a.gate = (const float*)gate; a.beta = (const float*)beta; a.head_decay = (const float*)head_decay;
    a.ldq = ldq; a.ldk = ldk; a.ldv = ldv;
    a.out = (float*)out; a.state = (float*)state; a.state_stride = state_stride;
    a.chunk_meta = (const int32_t*)chunk_meta; a.req_chunks = (const int32_t*)req_chunks;
    a.slots = (const int32_t*)slots; a.positions = (const int32_t*)positions;
    a.n_chunks = n_chunks; a.H = H; a.G = Gq; a.dk = dk; a.dv = dv;
    a.states = (float*)states; a.gain = (float*)gain; a.frag = (uint4*)frag; a.u = (float*)u;
    cudaStream_t s = (cudaStream_t)stream;
    if (dk <= 64) return dv <= 64 ? lc_run<64, 64>(a, n_requests, s) : lc_run<64, 128>(a, n_requests, s);
    return dv <= 64 ? lc_run<128, 64>(a, n_requests, s) : lc_run<128, 128>(a, n_requests, s);
}

template <int DK, int DV>
static int lc_run_forget(const LcArgs& a, int n_requests, cudaStream_t s) {
    const dim3 chunks(a.H, a.n_chunks);
    const size_t tile = LC_C * LC_LD * sizeof(float);
    if (const int rc = lc_launch<lc_forget_state_kernel<DK, DV>>(chunks, 256, 2 * tile, s, a)) return rc;
    const long long size = (long long)a.H * a.dv * a.dk;
    if (const int rc = lc_launch<lc_carry_kernel<true>>(dim3(ceil_div(size / 4, 256), n_requests), 256, 0, s, a)) return rc;
    return lc_launch<lc_forget_output_kernel<DK, DV>>(chunks, 256, 3 * tile, s, a);
}

// The recurrence with a forget gate per key channel: f [tokens, H dk] beside q; gain fp32 [chunks, H, dk]; the rest as above.
MM_EXPORT int mm_forget_gate_chunk(const void* q, const void* f, const void* v, int ldq, int ldf, int ldv, void* out, void* state,
                                   long long state_stride, const void* chunk_meta, const void* req_chunks, const void* slots,
                                   const void* positions, int n_requests, int n_chunks, int H, int dk, int dv, void* states, void* gain,
                                   void* stream) {
    MM_REQUIRE(H > 0, "forget gate chunks: bad sizes");
    MM_REQUIRE(mm_linear_chunk_supported(q, f, v, ldq, ldf, ldv, state, state_stride, dk, dv), "forget gate chunks: sizes or pointers that the products do not take");
    MM_REQUIRE(out && slots && positions && chunk_meta && req_chunks && states && gain, "forget gate chunks: the lists and the scratch are needed");
    MM_REQUIRE((((uintptr_t)out | (uintptr_t)states | (uintptr_t)gain) & 15) == 0, "forget gate chunks: the scratch starts on 16-byte boundaries");
    MM_REQUIRE(n_chunks <= 65535 && n_requests <= 65535, "forget gate chunks: too many chunks or requests");
    if (n_requests <= 0 || n_chunks <= 0) return MM_OK;
    LcArgs a = {};
    a.q = (const float*)q; a.k = (const float*)f; a.v = (const float*)v;
    a.ldq = ldq; a.ldk = ldf; a.ldv = ldv;
    a.out = (float*)out; a.state = (float*)state; a.state_stride = state_stride;
    a.chunk_meta = (const int32_t*)chunk_meta; a.req_chunks = (const int32_t*)req_chunks;
    a.slots = (const int32_t*)slots; a.positions = (const int32_t*)positions;
    a.n_chunks = n_chunks; a.H = a.G = H; a.dk = dk; a.dv = dv;
    a.states = (float*)states; a.gain = (float*)gain;
    cudaStream_t s = (cudaStream_t)stream;
    if (dk <= 64) return dv <= 64 ? lc_run_forget<64, 64>(a, n_requests, s) : lc_run_forget<64, 128>(a, n_requests, s);
    return dv <= 64 ? lc_run_forget<128, 64>(a, n_requests, s) : lc_run_forget<128, 128>(a, n_requests, s);
}
