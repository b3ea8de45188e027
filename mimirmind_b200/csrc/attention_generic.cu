// Paged causal attention with grouped KV heads, fp32 arithmetic, any head size.
//
// The plain form: one warp per (token, query head).  The key range of a token is cut into chunks of 32
// keys aligned to absolute position, and the running (max, sum, output) is updated
// chunk by chunk, so the result for a token depends only on its own position and keys:
// never on how the tokens were cut into steps or on what else is in the batch.  This is
// the kernel of the 32-bit path and the fallback of the bfloat16 path for head sizes the
// tensor-core kernels are not built for.
//
// Formula (reference src/compute/Attention.cpp:43-94): kv head g = (h*G)/H; a query at
// absolute position a sees keys [max(0, a+1-W), a] (W = 0: all); s_j = (q.k_j)*scale;
// p = softmax(s); o = sum_j p_j v_j.
//
// fp32 tensors of head size 64 or 128, the 32-bit path's own, take two kernels that do the same operations in the same
// order on tiles in shared memory (bit-equal to the plain form): `attention_tile_f32_kernel` for runs of consecutive tokens of one
// request, `attention_token_f32_kernel` for single tokens.  Both are launched; which of the two owns a row follows from its
// run alone (how many of the 32 rows of its tile belong to its request), so neither needs a list from the host.
#include "common.cuh"

#define ATT_MAX_ACC 16  // head_dim <= 512

template <typename T>
__global__ void attention_generic_kernel(const T* __restrict__ q, const T* __restrict__ k_pages,
                                         const T* __restrict__ v_pages, T* __restrict__ out,
                                         const int32_t* __restrict__ positions, const int32_t* __restrict__ token_req,
                                         const int32_t* __restrict__ block_table, int table_width, int page_size,
                                         int n_tokens, int H, int G, int hd, int window, float scale) {
    extern __shared__ float q_smem[];  // [warps][hd]
    const int warps_per_block = blockDim.x >> 5;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long item = (long long)blockIdx.x * warps_per_block + warp;
    if (item >= (long long)n_tokens * H) return;
    const int t = (int)(item / H), h = (int)(item - (long long)t * H);
    const int g = (h * G) / H;
    const int pos = positions[t];
    const int req = token_req[t];
    const int32_t* table = block_table + (size_t)req * table_width;
    const int hi = pos + 1;
    const int lo = (window > 0 && hi > window) ? hi - window : 0;

    float* qs = q_smem + warp * hd;
    const T* qrow = q + ((size_t)t * H + h) * hd;
    for (int d = lane; d < hd; d += 32) qs[d] = to_f32<T>(qrow[d]);
    __syncwarp();

    float m = -INFINITY, l = 0.0f;
    float acc[ATT_MAX_ACC];
#pragma unroll
    for (int a = 0; a < ATT_MAX_ACC; ++a) acc[a] = 0.0f;
    const size_t head_off = (size_t)g * page_size * hd;
    const size_t page_stride = (size_t)G * page_size * hd;

    for (int c = (lo / 32) * 32; c < hi; c += 32) {
        const int j = c + lane;
        const bool valid = (j >= lo) && (j < hi);
        float s = -INFINITY;
        if (valid) {
            const int page = table[j / page_size];
            const T* kr = k_pages + (size_t)page * page_stride + head_off + (size_t)(j % page_size) * hd;
            float dot = 0.0f;
            for (int d = 0; d < hd; ++d) dot = fmaf(qs[d], to_f32<T>(kr[d]), dot);
            s = dot * scale;
        }
        const float m_new = fmaxf(m, warp_max(s));
        const float alpha = expf(m - m_new);  // m = -inf on the first chunk gives 0
        const float p = valid ? expf(s - m_new) : 0.0f;
        l = l * alpha + warp_sum(p);
#pragma unroll
        for (int a = 0; a < ATT_MAX_ACC; ++a) acc[a] *= alpha;
        for (int jj = 0; jj < 32; ++jj) {
            const int key = c + jj;
            if (key < lo || key >= hi) continue;  // uniform over the warp
            const float pj = __shfl_sync(0xffffffffu, p, jj);
            const int page = table[key / page_size];
            const T* vr = v_pages + (size_t)page * page_stride + head_off + (size_t)(key % page_size) * hd;
#pragma unroll
            for (int a = 0; a < ATT_MAX_ACC; ++a) {
                const int d = a * 32 + lane;
                if (d < hd) acc[a] = fmaf(pj, to_f32<T>(vr[d]), acc[a]);
            }
        }
        m = m_new;
    }
    const float inv_l = (l > 0.0f) ? 1.0f / l : 0.0f;
    T* orow = out + ((size_t)t * H + h) * hd;
#pragma unroll
    for (int a = 0; a < ATT_MAX_ACC; ++a) {
        const int d = a * 32 + lane;
        if (d < hd) orow[d] = from_f32<T>(acc[a] * inv_l);
    }
}

// ---------------------------------------------------------------------------------------------------------------
// fp32, head sizes 64 and 128
// ---------------------------------------------------------------------------------------------------------------
#define ATT_TILE 32          // query rows of a tile, and keys of a chunk
#define ATT_RUN_MIN 4        // shorter runs go token by token

__device__ __forceinline__ void att_cp16(void* smem, const void* gmem, bool in) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(smem);
    const int bytes = in ? 16 : 0;               // 0: zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(gmem), "r"(bytes));
}
__device__ __forceinline__ void att_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void att_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// Where a key of the head stands in its pool; -1: not one that is read.
__device__ __forceinline__ long long att_offset(const int32_t* __restrict__ table, int key, int lo, int hi, int page_size, long long page_stride,
                                                long long head_off, int hd) {
    if (key < lo || key >= hi) return -1;
    return (long long)table[key / page_size] * page_stride + head_off + (long long)(key % page_size) * hd;
}

// A tile of 32 rows of one head, 128 threads: thread (ty, tx) owns the scores of rows 2 ty, 2 ty + 1 and keys tx, tx + 8, tx + 16, tx + 24 of
// a chunk, and the outputs of the same rows in the columns 32 g + 4 tx...  Bound by the chain of chunks and the latency of the
// shared-memory reads that feed the FMA units (a warp per scheduler at most tiles; one row a thread and eight warps read half as much again: 66 us), so what
// is multiplied next is read while the current numbers are multiplied; the next chunk's keys and values arrive under the current one, their places looked up two chunks ahead.
// The chunk's sum is added up in the order of a warp's butterfly over the key's place in the chunk: 16, 8 apart within a
// thread, 4, 2, 1 apart between the eight threads of a row.  Keys that a row does not see are skipped, not multiplied by zero.
// 509 tokens, 14 heads of 64: 51 us (without the reads ahead 59; a warp per token and head, the plain form: 820).
template <int HD>
__global__ void __launch_bounds__(128) attention_tile_f32_kernel(const float* __restrict__ q, const float* __restrict__ k_pages,
                                                                 const float* __restrict__ v_pages, float* __restrict__ out,
                                                                 const int32_t* __restrict__ positions, const int32_t* __restrict__ token_req,
                                                                 const int32_t* __restrict__ block_table, int table_width, int page_size,
                                                                 int n_tokens, int H, int G, int window, float scale) {
    constexpr int LD = HD + 4, LP = ATT_TILE + 4, CG = HD / 32, RP = 2;
    extern __shared__ __align__(16) float tile_smem[];
    float* sq = tile_smem;                       // [32][LD]
    float* sk = sq + ATT_TILE * LD;              // [2][32][LD]
    float* sv = sk + 2 * ATT_TILE * LD;          // [2][32][HD]
    float* sp = sv + 2 * ATT_TILE * HD;          // [32][LP]
    __shared__ long long soff[3][32];            // where the keys of three consecutive chunks stand
    const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3;
    const int h = blockIdx.x, g = (int)(((long long)h * G) / H);
    const int t0 = (int)(gridDim.y - 1 - blockIdx.y) * ATT_TILE;       // the longest tiles of a prompt first
    const int stop = min(n_tokens, t0 + ATT_TILE);
    const long long head_off = (long long)g * page_size * HD, page_stride = (long long)G * page_size * HD;

    for (int begin = t0; begin < stop;) {
        const int req = token_req[begin];
        int end = begin + 1;
        while (end < stop && token_req[end] == req) ++end;
        const int rows = end - begin, first = begin;
        begin = end;
        if (rows < ATT_RUN_MIN) continue;
        const int32_t* table = block_table + (size_t)req * table_width;
        int lo[RP], hi[RP], lo_all = 0x7fffffff, hi_all = 0;
#pragma unroll
        for (int i = 0; i < RP; ++i) {
            const int r = ty * RP + i;
            hi[i] = r < rows ? positions[first + r] + 1 : 0;
            lo[i] = (window > 0 && hi[i] > window) ? hi[i] - window : 0;
        }
        {
            const int r = tid & 31;
            const int top = r < rows ? positions[first + r] + 1 : 0;
            int low = r < rows ? ((window > 0 && top > window) ? top - window : 0) : 0x7fffffff;
            hi_all = __reduce_max_sync(0xffffffffu, top);
            lo_all = __reduce_min_sync(0xffffffffu, low);
        }
        const int c0 = lo_all / 32 * 32;
        __syncthreads();                         // the run before is through with the buffers
        if (tid < 64) soff[tid >> 5][tid & 31] = att_offset(table, c0 + tid, lo_all, hi_all, page_size, page_stride, head_off, HD);
        for (int idx = tid; idx < ATT_TILE * (HD / 4); idx += 128) {
            const int r = idx / (HD / 4), d = (idx % (HD / 4)) * 4;
            const bool in = r < rows;
            att_cp16(sq + r * LD + d, q + ((size_t)(first + (in ? r : 0)) * H + h) * HD + d, in);
        }
        __syncthreads();
        auto fill = [&](int n) {                 // chunk n
            float* dk = sk + (n & 1) * ATT_TILE * LD;
            float* dv = sv + (n & 1) * ATT_TILE * HD;
#pragma unroll
            for (int e = 0; e < ATT_TILE * (HD / 4) / 128; ++e) {
                const int idx = tid + e * 128, r = idx / (HD / 4), d = (idx % (HD / 4)) * 4;
                const long long off = soff[n % 3][r];
                const long long at = off < 0 ? 0 : off + d;
                att_cp16(dk + r * LD + d, k_pages + at, off >= 0);
                att_cp16(dv + r * HD + d, v_pages + at, off >= 0);
            }
            att_commit();
        };
        fill(0);
        float m[RP], l[RP], acc[RP][4 * CG];
#pragma unroll
        for (int i = 0; i < RP; ++i) {
            m[i] = -INFINITY;
            l[i] = 0.0f;
#pragma unroll
            for (int a = 0; a < 4 * CG; ++a) acc[i][a] = 0.0f;
        }
        int n = 0;
        for (int c = c0; c < hi_all; c += 32, ++n) {
            if (c + 32 < hi_all) {
                fill(n + 1);
                att_wait<1>();
            } else {
                att_wait<0>();
            }
            __syncthreads();
            if (tid < 32) soff[(n + 2) % 3][tid] = att_offset(table, c + 64 + tid, lo_all, hi_all, page_size, page_stride, head_off, HD);
            const float* kb = sk + (n & 1) * ATT_TILE * LD;
            const float* vb = sv + (n & 1) * ATT_TILE * HD;
            float s[RP][4];
#pragma unroll
            for (int i = 0; i < RP; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) s[i][j] = 0.0f;
            // the numbers of the next four columns are read while the current ones are multiplied
            auto scores = [&](float4* a, float4* b, int d) {
#pragma unroll
                for (int i = 0; i < RP; ++i) a[i] = *reinterpret_cast<const float4*>(sq + (ty * RP + i) * LD + d);
#pragma unroll
                for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(kb + (tx + 8 * j) * LD + d);
            };
            float4 qa[2][RP], ka[2][4];
            scores(qa[0], ka[0], 0);
#pragma unroll
            for (int d = 0; d < HD; d += 4) {
                const int u = (d >> 2) & 1;
                if (d + 4 < HD) scores(qa[u ^ 1], ka[u ^ 1], d + 4);
#define ATT_SCORE(C)                                       \
    _Pragma("unroll") for (int i = 0; i < RP; ++i)         \
        _Pragma("unroll") for (int j = 0; j < 4; ++j) s[i][j] = fmaf(qa[u][i].C, ka[u][j].C, s[i][j])
                ATT_SCORE(x);
                ATT_SCORE(y);
                ATT_SCORE(z);
                ATT_SCORE(w);
#undef ATT_SCORE
            }
            bool whole = true;                   // every row of the warp's sees every key of the chunk
#pragma unroll
            for (int i = 0; i < RP; ++i) {
                const int r = ty * RP + i;
                const bool any = lo[i] < c + 32 && hi[i] > c;          // the row sees keys of this chunk
                if (r < rows && !(lo[i] <= c && hi[i] >= c + 32)) whole = false;
                float p[4], top = -INFINITY;
                bool valid[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int key = c + tx + 8 * j;
                    valid[j] = key >= lo[i] && key < hi[i];
                    s[i][j] = valid[j] ? s[i][j] * scale : -INFINITY;
                    top = fmaxf(top, s[i][j]);
                }
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
                const float m_new = any ? fmaxf(m[i], top) : m[i];
                const float alpha = any ? expf(m[i] - m_new) : 1.0f;   // m = -inf on the first chunk gives 0
#pragma unroll
                for (int j = 0; j < 4; ++j) p[j] = valid[j] ? expf(s[i][j] - m_new) : 0.0f;
                float sum = (p[0] + p[2]) + (p[1] + p[3]);             // keys 16 apart, then 8 apart
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                if (any) {
                    l[i] = l[i] * alpha + sum;
                    m[i] = m_new;
#pragma unroll
                    for (int a = 0; a < 4 * CG; ++a) acc[i][a] *= alpha;
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) sp[r * LP + tx + 8 * j] = p[j];
            }
            whole = __all_sync(0xffffffffu, whole);
            __syncwarp();                        // a row's probabilities are written and read by the same eight threads
            if (whole) {
                auto values = [&](float4* v, int j) {
#pragma unroll
                    for (int a = 0; a < CG; ++a) v[a] = *reinterpret_cast<const float4*>(vb + j * HD + a * 32 + tx * 4);
                };
                float4 va[2][CG];
                values(va[0], 0);
#pragma unroll
                for (int j = 0; j < 32; j += 4) {
                    float4 p[RP];
#pragma unroll
                    for (int i = 0; i < RP; ++i) p[i] = *reinterpret_cast<const float4*>(sp + (ty * RP + i) * LP + j);
#pragma unroll
                    for (int jj = 0; jj < 4; ++jj) {
                        if (j + jj + 1 < 32) values(va[(jj + 1) & 1], j + jj + 1);
#pragma unroll
                        for (int a = 0; a < CG; ++a) {
                            const float4 v = va[jj & 1][a];
#pragma unroll
                            for (int i = 0; i < RP; ++i) {
                                const float pj = jj == 0 ? p[i].x : jj == 1 ? p[i].y : jj == 2 ? p[i].z : p[i].w;
                                acc[i][4 * a] = fmaf(pj, v.x, acc[i][4 * a]);
                                acc[i][4 * a + 1] = fmaf(pj, v.y, acc[i][4 * a + 1]);
                                acc[i][4 * a + 2] = fmaf(pj, v.z, acc[i][4 * a + 2]);
                                acc[i][4 * a + 3] = fmaf(pj, v.w, acc[i][4 * a + 3]);
                            }
                        }
                    }
                }
            } else {
#pragma unroll 4
                for (int j = 0; j < 32; ++j) {
                    const int key = c + j;
#pragma unroll
                    for (int a = 0; a < CG; ++a) {
                        const float4 v = *reinterpret_cast<const float4*>(vb + j * HD + a * 32 + tx * 4);
#pragma unroll
                        for (int i = 0; i < RP; ++i) {
                            const float pj = sp[(ty * RP + i) * LP + j];
                            if (key >= lo[i] && key < hi[i]) {
                                acc[i][4 * a] = fmaf(pj, v.x, acc[i][4 * a]);
                                acc[i][4 * a + 1] = fmaf(pj, v.y, acc[i][4 * a + 1]);
                                acc[i][4 * a + 2] = fmaf(pj, v.z, acc[i][4 * a + 2]);
                                acc[i][4 * a + 3] = fmaf(pj, v.w, acc[i][4 * a + 3]);
                            }
                        }
                    }
                }
            }
            __syncthreads();                     // before this buffer is filled again
        }
#pragma unroll
        for (int i = 0; i < RP; ++i) {
            const int r = ty * RP + i;
            if (r >= rows) continue;
            const float inv_l = (l[i] > 0.0f) ? 1.0f / l[i] : 0.0f;
            float* orow = out + ((size_t)(first + r) * H + h) * HD;
#pragma unroll
            for (int a = 0; a < CG; ++a)
                *reinterpret_cast<float4*>(orow + a * 32 + tx * 4) =
                    make_float4(acc[i][4 * a] * inv_l, acc[i][4 * a + 1] * inv_l, acc[i][4 * a + 2] * inv_l, acc[i][4 * a + 3] * inv_l);
        }
    }
}

// One token and head at a time per block of four warps (rows blockIdx.z, blockIdx.z + gridDim.z, ... of the tile blockIdx.y that stand in a
// short run): a segment of 128 keys at a time, a warp per chunk of 32.  The scores, chunk maxima and chunk sums of a segment are
// independent once the maxima before a chunk are known, so they are made side by side; what remains in order is a thread's chain
// of products over the keys in its column of the output.  Bound by that chain (4 clocks a key) and by the latency of a segment's
// copies: the next keys are requested when the scores are through, the next values after the chain, their places a segment ahead.
// 4 tokens, 301 keys, 14 heads of 64: 14 us (the plain form: 393; with a look into the page table per 16-byte copy: 23).
template <int HD>
__global__ void __launch_bounds__(128) attention_token_f32_kernel(const float* __restrict__ q, const float* __restrict__ k_pages,
                                                                  const float* __restrict__ v_pages, float* __restrict__ out,
                                                                  const int32_t* __restrict__ positions, const int32_t* __restrict__ token_req,
                                                                  const int32_t* __restrict__ block_table, int table_width, int page_size,
                                                                  int n_tokens, int H, int G, int window, float scale) {
    constexpr int LD = HD + 4, SEG = 128;
    extern __shared__ __align__(16) float token_smem[];
    float* sk = token_smem;                      // [128][LD]
    float* sv = sk + SEG * LD;                   // [128][HD]
    float* sq = sv + SEG * HD;                   // [HD]
    float* sp = sq + HD;                         // [128]
    __shared__ long long soff[2][SEG];
    __shared__ float chunk_max[4], chunk_sum[4];
    const int h = blockIdx.x, g = (int)(((long long)h * G) / H), t0 = blockIdx.y * ATT_TILE;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int lane_req = t0 + lane < n_tokens ? token_req[t0 + lane] : -1;
    const long long head_off = (long long)g * page_size * HD, page_stride = (long long)G * page_size * HD;
    for (int row = blockIdx.z; row < ATT_TILE && t0 + row < n_tokens; row += gridDim.z) {
        const int t = t0 + row, req = __shfl_sync(0xffffffffu, lane_req, row);
        {   // the length of the row's run: set bits that follow one another around the row's own
            const uint32_t same = __ballot_sync(0xffffffffu, lane_req == req);
            const uint32_t up = ~(same >> row), down = ~(same << (31 - row));
            const int run = (up ? __ffs(up) - 1 : 32) + (down ? __clz(down) : 32) - 1;
            if (run >= ATT_RUN_MIN) continue;    // the tile kernel's
        }
        const int32_t* table = block_table + (size_t)req * table_width;
        const int hi = positions[t] + 1, lo = (window > 0 && hi > window) ? hi - window : 0;
        const int c0 = lo / 32 * 32;
        __syncthreads();                         // the row before is through with the buffers
        soff[0][tid] = att_offset(table, c0 + tid, lo, hi, page_size, page_stride, head_off, HD);
        if (tid < HD / 4) *reinterpret_cast<float4*>(sq + tid * 4) = *reinterpret_cast<const float4*>(q + ((size_t)t * H + h) * HD + tid * 4);
        __syncthreads();
        auto fill = [&](const float* __restrict__ pages, float* dst, int ld, int n) {
#pragma unroll
            for (int e = 0; e < SEG * (HD / 4) / 128; ++e) {
                const int idx = tid + e * 128, r = idx / (HD / 4), d = (idx % (HD / 4)) * 4;
                const long long off = soff[n & 1][r];
                att_cp16(dst + r * ld + d, pages + (off < 0 ? 0 : off + d), off >= 0);
            }
            att_commit();
        };
        fill(k_pages, sk, LD, 0);
        fill(v_pages, sv, HD, 0);
        float m = -INFINITY, l = 0.0f, acc = 0.0f;
        int n = 0;
        for (int base = c0; base < hi; base += SEG, ++n) {
            const bool more = base + SEG < hi;
            if (more) soff[(n + 1) & 1][tid] = att_offset(table, base + SEG + tid, lo, hi, page_size, page_stride, head_off, HD);
            att_wait<1>();                       // this segment's keys (its values may still be on their way)
            __syncthreads();
            const int key = base + tid;
            const bool valid = key >= lo && key < hi;
            float s = -INFINITY;
            {
                float dot = 0.0f;
                const float* kr = sk + tid * LD;
#pragma unroll 16
                for (int d = 0; d < HD; d += 4) {
                    const float4 a = *reinterpret_cast<const float4*>(sq + d), b = *reinterpret_cast<const float4*>(kr + d);
                    dot = fmaf(a.x, b.x, dot);
                    dot = fmaf(a.y, b.y, dot);
                    dot = fmaf(a.z, b.z, dot);
                    dot = fmaf(a.w, b.w, dot);
                }
                if (valid) s = dot * scale;
            }
            const float top = warp_max(s);
            if (lane == 0) chunk_max[warp] = top;
            __syncthreads();                     // also: every warp is through with the keys
            if (more) fill(k_pages, sk, LD, n + 1);
            else att_commit();
            const int chunks = min(4, (hi - base + 31) / 32);
            float mine = m;
            for (int w = 0; w <= warp; ++w) mine = fmaxf(mine, chunk_max[w]);
            const float p = valid ? expf(s - mine) : 0.0f;
            const float sum = warp_sum(p);
            sp[tid] = p;
            if (lane == 0) chunk_sum[warp] = sum;
            att_wait<1>();                       // the values
            __syncthreads();
            for (int w = 0; w < chunks; ++w) {
                const float m_new = fmaxf(m, chunk_max[w]);
                const float alpha = expf(m - m_new);  // m = -inf on the first chunk gives 0
                l = l * alpha + chunk_sum[w];
                m = m_new;
                if (tid < HD) {
                    acc *= alpha;
                    const int a = max(lo - (base + 32 * w), 0), b = min(hi - (base + 32 * w), 32);
                    const float* vr = sv + (32 * w) * HD + tid;
                    if (a == 0 && b == 32) {
#pragma unroll
                        for (int j = 0; j < 32; j += 4) {
                            const float4 pj = *reinterpret_cast<const float4*>(sp + 32 * w + j);
                            acc = fmaf(pj.x, vr[j * HD], acc);
                            acc = fmaf(pj.y, vr[(j + 1) * HD], acc);
                            acc = fmaf(pj.z, vr[(j + 2) * HD], acc);
                            acc = fmaf(pj.w, vr[(j + 3) * HD], acc);
                        }
                    } else {
                        for (int j = a; j < b; ++j) acc = fmaf(sp[32 * w + j], vr[j * HD], acc);
                    }
                }
            }
            __syncthreads();                     // before the values, the probabilities and the chunks' numbers are replaced
            if (more) fill(v_pages, sv, HD, n + 1);
            else att_commit();
        }
        if (tid < HD) out[((size_t)t * H + h) * HD + tid] = acc * ((l > 0.0f) ? 1.0f / l : 0.0f);
    }
}

template <int HD>
static int launch_attention_f32(const void* q, const void* k_pages, const void* v_pages, void* out, const void* positions, const void* token_req,
                                const void* block_table, int table_width, int page_size, int n_tokens, int H, int G, int window, float scale,
                                cudaStream_t s) {
    const int tile_bytes = (ATT_TILE * (HD + 4) * 3 + 2 * ATT_TILE * HD + ATT_TILE * (ATT_TILE + 4)) * (int)sizeof(float);
    const int token_bytes = (128 * (HD + 4) + 128 * HD + HD + 128) * (int)sizeof(float);
    if (!mm_allow_smem<attention_tile_f32_kernel<HD>>(tile_bytes) || !mm_allow_smem<attention_token_f32_kernel<HD>>(token_bytes)) {
        mm_set_last_error("attention: cannot reserve shared memory");
        return MM_ERR_LAUNCH;
    }
    // Blocks of the token kernel per tile and head: one per row while that fills the GPU, fewer for a long step, where most rows are
    // the tile kernel's (a 509-token prompt with a block per row spent 39 us on blocks that found nothing to do).
    const int tiles = ceil_div(n_tokens, ATT_TILE);
    int per_tile = (int)(1024 / ((long long)H * tiles));
    per_tile = per_tile < 1 ? 1 : per_tile > ATT_TILE ? ATT_TILE : per_tile;
    if (per_tile > n_tokens) per_tile = n_tokens;
    mm_launch(attention_token_f32_kernel<HD>, dim3(H, tiles, per_tile), dim3(128), (size_t)token_bytes, s, (const float*)q, (const float*)k_pages,
              (const float*)v_pages, (float*)out, (const int32_t*)positions, (const int32_t*)token_req, (const int32_t*)block_table, table_width,
              page_size, n_tokens, H, G, window, scale);
    MM_CHECK_LAUNCH();
    if (n_tokens >= ATT_RUN_MIN) {
        mm_launch(attention_tile_f32_kernel<HD>, dim3(H, tiles), dim3(128), (size_t)tile_bytes, s, (const float*)q, (const float*)k_pages,
                  (const float*)v_pages, (float*)out, (const int32_t*)positions, (const int32_t*)token_req, (const int32_t*)block_table,
                  table_width, page_size, n_tokens, H, G, window, scale);
        MM_CHECK_LAUNCH();
    }
    return MM_OK;
}

MM_EXPORT int mm_attention_generic(const void* q, const void* k_pages, const void* v_pages, void* out, int dtype,
                                   const void* positions, const void* token_req, const void* block_table,
                                   int table_width, int page_size, int n_tokens, int H, int G, int hd, int window,
                                   float scale, void* stream) {
    MM_REQUIRE(n_tokens >= 0 && H > 0 && G > 0 && hd > 0 && H % G == 0, "attention: heads must be a positive multiple of kv heads");
    MM_REQUIRE(hd <= 32 * ATT_MAX_ACC, "attention: head_dim above 512 is not supported");
    MM_REQUIRE(page_size > 0 && table_width > 0 && window >= 0, "attention: bad page geometry or window");
    if (n_tokens == 0) return MM_OK;
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == MM_F32 && (hd == 64 || hd == 128) && ceil_div(n_tokens, ATT_TILE) <= 65535 &&
        (((uintptr_t)q | (uintptr_t)k_pages | (uintptr_t)v_pages | (uintptr_t)out) & 15) == 0) {
        return hd == 64 ? launch_attention_f32<64>(q, k_pages, v_pages, out, positions, token_req, block_table, table_width, page_size, n_tokens, H,
                                                   G, window, scale, s)
                        : launch_attention_f32<128>(q, k_pages, v_pages, out, positions, token_req, block_table, table_width, page_size, n_tokens, H,
                                                    G, window, scale, s);
    }
    const int warps = 4;
    const size_t smem = (size_t)warps * hd * sizeof(float);
    const long long items = (long long)n_tokens * H;
    const int blocks = (int)((items + warps - 1) / warps);
    if (dtype == MM_F32)
        attention_generic_kernel<float><<<blocks, warps * 32, smem, s>>>(
            (const float*)q, (const float*)k_pages, (const float*)v_pages, (float*)out, (const int32_t*)positions,
            (const int32_t*)token_req, (const int32_t*)block_table, table_width, page_size, n_tokens, H, G, hd, window, scale);
    else if (dtype == MM_BF16)
        attention_generic_kernel<__nv_bfloat16><<<blocks, warps * 32, smem, s>>>(
            (const __nv_bfloat16*)q, (const __nv_bfloat16*)k_pages, (const __nv_bfloat16*)v_pages, (__nv_bfloat16*)out,
            (const int32_t*)positions, (const int32_t*)token_req, (const int32_t*)block_table, table_width, page_size,
            n_tokens, H, G, hd, window, scale);
    else
        MM_REQUIRE(false, "attention: dtype must be float32 or bfloat16");
    MM_CHECK_LAUNCH();
    return MM_OK;
}
