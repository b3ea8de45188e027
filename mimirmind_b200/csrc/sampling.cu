// Device-side sampling over fp32 logits [R, V]: argmax, and temperature / top-k / top-p
// draws (one thread-block cluster per row, the CTAs of a cluster share the row), so no logits
// leave the GPU.
//
// Semantics follow the reference's host sampler (src/compute/Sampling.cpp:119-264):
//   * temperature <= 0 or top_k == 1 is greedy; greedy is the first strict maximum,
//     i.e. the lowest index among equal maxima (:14-27; kernels/cuda/llm/argmax_rows.cu).
//   * otherwise p_i = exp(l_i/T - max/T); candidates are ordered by logit descending;
//     top-k keeps the k best; top-p keeps the smallest prefix whose share of the kept
//     mass reaches p; one uniform u picks the first candidate whose cumulative
//     probability exceeds u.
//   * optional before that: soft-cap cap*tanh(l/cap) (:38-44), then repetition /
//     frequency / presence penalties over a window of recent tokens (:66-117).
// Differences, by design: the order is found with a radix select instead of a sort;
// probabilities are summed as 40-bit fixed-point integers so that the result does not
// depend on the order in which threads add them; equal logits are ordered by index, and
// a top-k or top-p cut that falls inside a run of equal logits keeps the whole run (the
// reference's sort leaves that order unspecified).  The uniform number comes from a
// counter-based generator keyed by (seed, draw index) per request, so a request's stream
// does not depend on what else is in the batch.
#include "common.cuh"

#define SAMPLE_THREADS 1024     // of the whole-row argmax
#define FIXED_ONE 1099511627776.0f  // 2^40

__device__ __forceinline__ uint32_t order_key(float v) {
    // (u | 0x80000000 would be compiled to a negation of the absolute value, which does not keep a NaN's bits)
    const uint32_t u = __float_as_uint(v);
    return u ^ ((uint32_t)((int32_t)u >> 31) | 0x80000000u);
}
// The key among masses: a NaN counts as one of the best for top-k, but stands below all positive logits where masses are added up.
__device__ __forceinline__ uint32_t mass_key(float v) {
    const uint32_t key = order_key(v);
    return key > 0xff800000u ? 0x7fffffffu : key;
}

// splitmix64 finaliser over (seed, counter): a stateless stream of 64-bit numbers
__host__ __device__ __forceinline__ uint64_t mix64(uint64_t seed, uint64_t counter) {
    uint64_t z = seed + 0x9E3779B97F4A7C15ull * (counter + 1);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

struct ArgmaxPair {
    float v;
    int i;
};

__device__ __forceinline__ ArgmaxPair better(ArgmaxPair a, ArgmaxPair b) {
    if (b.v > a.v || (b.v == a.v && b.i < a.i)) return b;
    return a;
}

__device__ int block_argmax(const float* __restrict__ row, int V, float* max_out) {
    __shared__ ArgmaxPair red[32];
    ArgmaxPair best{-INFINITY, 0x7fffffff};
    for (int i = threadIdx.x; i < V; i += blockDim.x) {
        const float v = row[i];
        if (v > best.v || (v == best.v && i < best.i)) best = ArgmaxPair{v, i};
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        ArgmaxPair other{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)};
        best = better(best, other);
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) red[warp] = best;
    __syncthreads();
    if (warp == 0) {
        ArgmaxPair b = (lane < (int)(blockDim.x >> 5)) ? red[lane] : ArgmaxPair{-INFINITY, 0x7fffffff};
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            ArgmaxPair other{__shfl_xor_sync(0xffffffffu, b.v, o), __shfl_xor_sync(0xffffffffu, b.i, o)};
            b = better(b, other);
        }
        if (lane == 0) red[0] = b;
    }
    __syncthreads();
    const ArgmaxPair r = red[0];
    if (max_out) *max_out = r.v;
    // a row of NaN or -inf only: every comparison failed, fall back to index 0
    return r.i == 0x7fffffff ? 0 : r.i;
}

__global__ void argmax_rows_kernel(const float* __restrict__ logits, int32_t* __restrict__ out, int V) {
    const float* row = logits + (size_t)blockIdx.x * V;
    const int idx = block_argmax(row, V, nullptr);
    if (threadIdx.x == 0) out[blockIdx.x] = idx;
}

MM_EXPORT int mm_argmax_rows(const void* logits, void* out, int R, int V, void* stream) {
    MM_REQUIRE(R >= 0 && V > 0, "argmax: bad sizes");
    if (R == 0) return MM_OK;
    mm_launch(argmax_rows_kernel, dim3(R), dim3(SAMPLE_THREADS), 0, (cudaStream_t)stream, (const float*)logits, (int32_t*)out, V);
    MM_CHECK_LAUNCH();
    return MM_OK;
}

// Two stages for wide rows: P blocks per row find (max, lowest index) of their slice, then one
// block per row reduces the P pairs.  `part` holds R*P pairs of (float value, int index).
__global__ void argmax_partial_kernel(const float* __restrict__ logits, float* __restrict__ part_val,
                                      int32_t* __restrict__ part_idx, int V, int P) {
    const int r = blockIdx.y, p = blockIdx.x;
    const int chunk = (V + P - 1) / P;
    const int begin = p * chunk, end = min(V, begin + chunk);
    const float* row = logits + (size_t)r * V;
    __shared__ ArgmaxPair red[32];
    ArgmaxPair best{-INFINITY, 0x7fffffff};
    for (int i = begin + threadIdx.x; i < end; i += blockDim.x) {
        const float v = row[i];
        if (v > best.v || (v == best.v && i < best.i)) best = ArgmaxPair{v, i};
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        ArgmaxPair other{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)};
        best = better(best, other);
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) red[warp] = best;
    __syncthreads();
    if (warp == 0) {
        ArgmaxPair b = (lane < (int)(blockDim.x >> 5)) ? red[lane] : ArgmaxPair{-INFINITY, 0x7fffffff};
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            ArgmaxPair other{__shfl_xor_sync(0xffffffffu, b.v, o), __shfl_xor_sync(0xffffffffu, b.i, o)};
            b = better(b, other);
        }
        if (lane == 0) {
            part_val[(size_t)r * P + p] = b.v;
            part_idx[(size_t)r * P + p] = b.i;
        }
    }
}

__global__ void argmax_final_kernel(const float* __restrict__ part_val, const int32_t* __restrict__ part_idx,
                                    int32_t* __restrict__ out, int P) {
    const int r = blockIdx.x, lane = threadIdx.x;
    ArgmaxPair best{-INFINITY, 0x7fffffff};
    for (int p = lane; p < P; p += 32) best = better(best, ArgmaxPair{part_val[(size_t)r * P + p], part_idx[(size_t)r * P + p]});
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        ArgmaxPair other{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)};
        best = better(best, other);
    }
    if (lane == 0) out[r] = best.i == 0x7fffffff ? 0 : best.i;
}

MM_EXPORT int mm_argmax_rows_split(const void* logits, void* out, void* part_val, void* part_idx, int R, int V, int P,
                                   void* stream) {
    MM_REQUIRE(R >= 0 && V > 0 && P >= 1 && P <= 1024 && R <= 65535, "argmax: bad sizes");
    if (R == 0) return MM_OK;
    cudaStream_t s = (cudaStream_t)stream;
    mm_launch(argmax_partial_kernel, dim3(P, R), dim3(256), 0, s, (const float*)logits, (float*)part_val, (int32_t*)part_idx, V, P);
    MM_CHECK_LAUNCH();
    mm_launch(argmax_final_kernel, dim3(R), dim3(32), 0, s, (const float*)part_val, (const int32_t*)part_idx, (int32_t*)out, P);
    MM_CHECK_LAUNCH();
    return MM_OK;
}

// ---- sampling: one thread-block cluster per row -------------------------------------------------------------
// The CTAs of a cluster take contiguous slices of the row.  Whatever the whole row decides (its maximum, the mass
// of the kept set, a histogram, how many elements carry the chosen key) is computed per CTA, published in shared
// memory, and read by every CTA of the cluster from its peers through distributed shared memory after one cluster
// barrier; all CTAs then hold the same numbers and take the same branch.  Publications alternate between two
// buffers, so one barrier per exchange is enough: a CTA can run at most one exchange ahead of a peer that is still
// reading.
//
// Top-k, top-p and the draw each look for one element of the same order (logit descending, index ascending): the first
// whose cumulative count or mass exceeds a target.  A row is read once from memory, 16 bytes a load, and kept in shared memory:
//   1. mass and count per eighth of a nat below the maximum (256 bins), in 16 copies that the lanes of a warp share out: a
//      warp's additions then hardly ever meet in a bank.  Masses in halves of 20 bits: shared memory adds 32-bit numbers by
//      itself, 64-bit ones by compare and swap.
//   2. From these each search's bin is known, or a short range of bins: top-p's target depends on what top-k keeps and the
//      draw's on what top-p keeps, which lies between the sums before and after a bin; all steps are monotone.
//   3. If more than DRAW_LIST numbers lie in these bins: the same once more with 1/2048 of a nat, over their numbers only.
//   4. The numbers of the bins go into a list, and the first CTA finds all three elements there.
// Bound by instructions (an exponential, three additions in shared memory and some 30 more per number, 75 numbers a thread) and
// by four or five exchanges of the cluster.  With a pass, two cluster barriers and a list for each search, and copies of the
// bins by warp, 32 rows of 152,064 logits with top-p took 62 us, this takes 44 (with 1.5 as temperature, where the cut
// lies among most of the row, 77 and 46; both from HBM).  The numbers in registers instead of shared memory, unrolled, took twice as long as
// before: 76 copies of a pass are more instructions than their cache holds.  So did bins of two nats in a column per thread,
// without atomics: what is saved there is lost on the second pass that they need.
// Rows with a NaN or an infinite maximum, and searches that end in more than DRAW_LIST logits within 1/2048 nat, take
// the radix select, four passes per search over the slice.
#define DRAW_THREADS 512
#define DRAW_WARPS (DRAW_THREADS / 32)
#define DRAW_COPIES 8                              // the radix select's histograms of a CTA: two warps share one
#define DRAW_LANES 16                              // copies of the bins: two lanes of a warp share one
#define DRAW_LIST 2048
#define DRAW_NEAR 512                              // numbers that a warp keeps the places of
#define DRAW_SLOTS 4                               // bins that are cut finer at once
#define DRAW_FINE (DRAW_SLOTS * 256)
#define DRAW_FEW 128                               // elements among which every one is compared with every other
#define DRAW_LO_MAX 3800                           // numbers of one bin whose low and high halves 32 bits hold: at most 2^20 e^(1/16) each
#define DRAW_ROOM 38016                            // numbers of a slice kept in shared memory beside the rest: 227 KB together
#define DRAW_SEGMENT (DRAW_LANES * DRAW_LO_MAX)    // numbers that the bins' sums have room for: longer slices go in segments
#define SAMPLE_MAX_CLUSTER 8

struct BinPlace {
    unsigned long long before, carry;              // the mass of the bins before it, what is left of the target
    unsigned long long upto;                       // the mass including it
    int bin, sub;                                  // sub: -1 without the finer bins
    uint32_t count;                                // numbers in it
};
struct BinTable {                                  // 256 bins: mass, count and their sums up to and including a bin
    unsigned long long mass[256], upto[256];
    uint32_t ct[256], upto_ct[256];
};

struct alignas(16) SampleShared {
    union {
        struct {
            uint32_t lo[257][DRAW_LANES], hi[257][DRAW_LANES], ct[257][DRAW_LANES];
        } hist;
        struct {
            union {
                struct {
                    uint32_t lo[DRAW_FINE], hi[DRAW_FINE];
                    unsigned long long pub[DRAW_FINE];             // the masses as published
                };
                unsigned long long own[DRAW_LIST];                 // then this CTA's candidates
                unsigned long long sublist[DRAW_LIST];             // then, in the first CTA, those of one bin
            };
            union {
                uint32_t ct[DRAW_FINE];                            // published
                struct {
                    uint32_t lo[256], hi[256], ct[256];
                } cut;                                             // then a cut within the list
            };
            BinTable tab[DRAW_SLOTS];                              // the cluster's
        } fine;
        unsigned long long whist[DRAW_COPIES][256];                // the radix select's
        int counts[DRAW_THREADS];
    };
    union {
        unsigned short near[DRAW_WARPS][DRAW_NEAR];                // places in the slice of the numbers of the bins that hold places, by warp
        unsigned long long list[DRAW_LIST];        // then, in the first CTA, the cluster's candidates: (order key << 32) | index
    };
    BinTable tab;                                  // the cluster's bins
    union {
        uint32_t pub_ct[256];
        unsigned long long few_w[DRAW_FEW];        // masses of a bin's candidates
    };
    union {
        struct {
            unsigned long long pub[2][256 + 4];    // what this CTA publishes: masses, or scalars in [256..]
            unsigned long long tot[256];           // of the radix select: the cluster's histogram
        };
        BinTable cut_tab;                          // of a cut within the list
    };
    unsigned long long warp_part[DRAW_WARPS];
    unsigned long long carry, before;              // what is left of the target inside the chosen bin; the mass of the bins before it
    unsigned long long found_mass;
    BinPlace place[2];
    float want[3][2];                              // where the searches may end, in 1/2048 nat below the maximum: from, up to
    uint32_t found_key, found_index, found_tie;
    uint32_t chosen, chosen_ct;
    uint32_t mask[8];                              // the bins that hold these places
    int slot_bin[DRAW_SLOTS];                      // those that are cut finer
    unsigned char slot_of[256], marked[257];       // a bin's slot + 1 (0: not cut); 1 for a bin that held places at first
    uint32_t n_list, list_n, few_n, too_many, is_fine;
    uint32_t range[2];
    int result;
};
static_assert(sizeof(SampleShared) % 16 == 0 && sizeof(SampleShared) + DRAW_ROOM * sizeof(float) <= 227 * 1024, "beyond a CTA's shared memory");

// This CTA's.  Functions that are called rather than inlined take it from here: a pointer that is passed to them would make every access of theirs,
// the atomic ones above all, one to an address of unknown kind.
__device__ __forceinline__ SampleShared* draw_shared() {
    extern __shared__ __align__(16) unsigned char sample_smem[];
    return reinterpret_cast<SampleShared*>(sample_smem);
}

struct ClusterCtx {
    const float* vals;                             // this CTA's slice: its copy in shared memory, or the row itself
    int vals_begin;                                // index of vals[0] in the row
    uint32_t rank, n_ranks;
    uint32_t round;                                // exchanges so far: selects the publication buffer
};

__device__ __forceinline__ void sample_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\n" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;\n" ::: "memory");
}
__device__ __forceinline__ uint32_t peer_address(const void* local, uint32_t rank) {
    const uint32_t addr = (uint32_t)__cvta_generic_to_shared(local);
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(remote) : "r"(addr), "r"(rank));
    return remote;
}
__device__ __forceinline__ unsigned long long ld_peer_u64(const unsigned long long* local, uint32_t rank) {
    unsigned long long v;
    asm volatile("ld.shared::cluster.u64 %0, [%1];\n" : "=l"(v) : "r"(peer_address(local, rank)) : "memory");
    return v;
}
// The same word of every CTA of the cluster: the loads go out together (a loop that adds each value as it arrives would
// wait for one remote load after the other).  v[r] for r >= n_ranks is 0.
__device__ __forceinline__ void ld_all_peers_u64(const unsigned long long* local, uint32_t n_ranks, unsigned long long* v) {
    uint32_t remote[SAMPLE_MAX_CLUSTER];
#pragma unroll
    for (uint32_t r = 0; r < SAMPLE_MAX_CLUSTER; ++r) remote[r] = peer_address(local, r < n_ranks ? r : 0u);
#pragma unroll
    for (uint32_t r = 0; r < SAMPLE_MAX_CLUSTER; ++r) {
        v[r] = 0ull;
        if (r < n_ranks) asm volatile("ld.shared::cluster.u64 %0, [%1];\n" : "=l"(v[r]) : "r"(remote[r]) : "memory");
    }
}
__device__ __forceinline__ uint32_t sum_all_peers_u32(const uint32_t* local, uint32_t n_ranks) {
    uint32_t remote[SAMPLE_MAX_CLUSTER], sum = 0;
#pragma unroll
    for (uint32_t r = 0; r < SAMPLE_MAX_CLUSTER; ++r) remote[r] = peer_address(local, r < n_ranks ? r : 0u);
    uint32_t v[SAMPLE_MAX_CLUSTER];
#pragma unroll
    for (uint32_t r = 0; r < SAMPLE_MAX_CLUSTER; ++r) {
        v[r] = 0u;
        if (r < n_ranks) asm volatile("ld.shared::cluster.u32 %0, [%1];\n" : "=r"(v[r]) : "r"(remote[r]) : "memory");
    }
#pragma unroll
    for (uint32_t r = 0; r < SAMPLE_MAX_CLUSTER; ++r) sum += v[r];
    return sum;
}
__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ unsigned long long warp_max_u64(unsigned long long v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, v, o);
        v = other > v ? other : v;
    }
    return v;
}

// Every CTA's value is reduced over its threads and published; returns the sum (or the maximum) over the cluster, the
// same in every thread of every CTA.
__device__ __noinline__ unsigned long long cluster_combine(ClusterCtx& c, unsigned long long mine, bool take_max) {
    SampleShared* sh = draw_shared();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    mine = take_max ? warp_max_u64(mine) : warp_sum_u64(mine);
    __syncthreads();
    if (lane == 0) sh->warp_part[warp] = mine;
    __syncthreads();
    const uint32_t b = c.round & 1;
    if (warp == 0) {
        unsigned long long v = lane < DRAW_WARPS ? sh->warp_part[lane] : 0ull;
        v = take_max ? warp_max_u64(v) : warp_sum_u64(v);
        if (lane == 0) sh->pub[b][256] = v;
    }
    __syncthreads();
    sample_cluster_sync();
    unsigned long long all = 0ull, v[SAMPLE_MAX_CLUSTER];
    ld_all_peers_u64(&sh->pub[b][256], c.n_ranks, v);
#pragma unroll
    for (uint32_t r = 0; r < SAMPLE_MAX_CLUSTER; ++r) all = take_max ? (v[r] > all ? v[r] : all) : all + v[r];
    ++c.round;
    return all;
}

__device__ __forceinline__ unsigned long long weight_of(float logit, float inv_t, float max_scaled) {
    const float p = expf(logit * inv_t - max_scaled);
    return (unsigned long long)(p * FIXED_ONE);
}
// The same of a plain row, whose weights are below 2^41, in halves of 20 bits (and what is above): by sums that cut off what lies below the integer.
struct Halves {
    uint32_t low, high;
};
__device__ __forceinline__ Halves weight_halves(float logit, float inv_t, float max_scaled) {
    const float p = expf(__fmaf_rn(logit, inv_t, -max_scaled));
    const float high = __fmaf_rz(p, 1048576.0f, 8388608.0f);
    const float low = __fadd_rz(__fmaf_rn(high - 8388608.0f, -1048576.0f, p * FIXED_ONE), 8388608.0f);
    return Halves{__float_as_uint(low) & 0x7fffffu, __float_as_uint(high) & 0x7fffffu};
}
__device__ __forceinline__ unsigned long long weight_below(float logit, float inv_t, float max_scaled) {
    const Halves w = weight_halves(logit, inv_t, max_scaled);
    return ((unsigned long long)w.high << 20) + w.low;
}
__device__ __forceinline__ float logit_of_key(uint32_t key) {
    return __uint_as_float((key & 0x80000000u) ? (key & 0x7fffffffu) : ~key);
}

// The bin of tot (in ascending order of bins) in which the cumulative weight exceeds `target`, by the first warp: left in
// chosen, with what is left of the target in carry.  A target at or beyond the total (rounding at the tail) takes the last bin
// that holds anything.
__device__ __noinline__ void pick_bin(unsigned long long target) {
    SampleShared* sh = draw_shared();
    __syncthreads();
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        unsigned long long h[8], mine = 0ull;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            h[j] = sh->tot[8 * lane + j];
            mine += h[j];
        }
        unsigned long long incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long up = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += up;
        }
        unsigned long long cum = incl - mine, rem = 0ull, last_rem = 0ull;
        int chosen = -1, last = -1;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (chosen < 0 && h[j] && target < cum + h[j]) {
                chosen = 8 * lane + j;
                rem = target - cum;
            }
            if (h[j]) {
                last = 8 * lane + j;
                last_rem = h[j] - 1ull;
            }
            cum += h[j];
        }
        const uint32_t found = __ballot_sync(0xffffffffu, chosen >= 0), any = __ballot_sync(0xffffffffu, last >= 0);
        const int owner = found ? __ffs(found) - 1 : any ? 31 - __clz(any) : 0;
        if (lane == owner) {
            sh->chosen = (uint32_t)(found ? chosen : last < 0 ? 0 : last);
            sh->carry = found ? rem : last_rem;
        }
    }
    __syncthreads();
}

// The sums of a table, by one warp: eight rows of 32 bins side by side.
__device__ __noinline__ void sum_table(uint32_t offset) {     // of the table within SampleShared
    BinTable* t = reinterpret_cast<BinTable*>(reinterpret_cast<unsigned char*>(draw_shared()) + offset);
    const int lane = threadIdx.x & 31;
    unsigned long long m[8], carry = 0ull;
    uint32_t n[8], carry_ct = 0u;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        m[j] = t->mass[32 * j + lane];
        n[j] = t->ct[32 * j + lane];
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const unsigned long long up = __shfl_up_sync(0xffffffffu, m[j], o);
            const uint32_t up_ct = __shfl_up_sync(0xffffffffu, n[j], o);
            if (lane >= o) {
                m[j] += up;
                n[j] += up_ct;
            }
        }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        t->upto[32 * j + lane] = m[j] + carry;
        t->upto_ct[32 * j + lane] = n[j] + carry_ct;
        carry += __shfl_sync(0xffffffffu, m[j], 31);
        carry_ct += __shfl_sync(0xffffffffu, n[j], 31);
    }
}

// Bins of a plain row, monotone in the logit (a rounded product and sum, a scaling and limits are): 65536 of 1/2048 nat below the
// maximum, the last one without an end; 256 of them are a bin of the first level.  Both come from one rounded number, the distance from the maximum
// in 32 nats, by powers of two, so that a logit's bin of the first level holds its finer one whatever the temperature (near 1e38
// inv_t / 32 is below the normal numbers and not what inv_t is).
struct DrawBins {
    float inv_t, max_scaled, inv_t32, max_scaled32;                // as they are, and divided by 32
    __device__ __forceinline__ float below(float v) const { return __saturatef(__fmaf_rn(-v, inv_t32, max_scaled32)); }
    __device__ __forceinline__ float place(float v) const { return fminf(65536.0f * below(v), 65535.0f); }
    // The bin of the first level, 0 to 256 (256 is the end of bin 255), as the low bits of the result: the limits come with the sum, so this is
    // two instructions.
    __device__ __forceinline__ uint32_t first_bits(float v) const { return __float_as_uint(__fmaf_rz(below(v), 256.0f, 8388608.0f)); }
    // the integer part, from the low bits of a sum that cuts the rest off
    __device__ __forceinline__ int of(float v) const { return (int)(__float_as_uint(__fadd_rz(place(v), 8388608.0f)) & 65535u); }
};

// the q-th four numbers of a slice from memory; what lies beyond its end is -inf
__device__ __forceinline__ float4 slice_quad(const float* __restrict__ slice, int len, int vec, int q) {
    float4 w = make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
    const float* at = slice + 4 * q;
    if (vec) return 4 * q < len ? __ldg(reinterpret_cast<const float4*>(at)) : w;
    if (4 * q < len) w.x = __ldg(at);
    if (4 * q + 1 < len) w.y = __ldg(at + 1);
    if (4 * q + 2 < len) w.z = __ldg(at + 2);
    if (4 * q + 3 < len) w.w = __ldg(at + 3);
    return w;
}
// four numbers of a plain row into this lane's copy of the bins of the first level
__device__ __forceinline__ void add_to_bins(const float4& four, const DrawBins& bins) {
    SampleShared* sh = draw_shared();
    // a bin's word for this lane: 64 bytes a bin, the exponent of first_bits shifted out by the start
    const uint32_t cell = (uint32_t)__cvta_generic_to_shared(&sh->hist.lo[0][threadIdx.x % DRAW_LANES]) - (0x4b000000u * 64u);
    constexpr uint32_t HI = sizeof(sh->hist.lo), CT = 2 * sizeof(sh->hist.lo);
    const float x[4] = {four.x, four.y, four.z, four.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const Halves w = weight_halves(x[j], bins.inv_t, bins.max_scaled);
        const uint32_t at = bins.first_bits(x[j]) * 64u + cell;
        asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(at), "r"(w.low) : "memory");
        if (w.high) asm volatile("red.shared.add.u32 [%0+%2], %1;" ::"r"(at), "r"(w.high), "n"(HI) : "memory");
        asm volatile("red.shared.add.u32 [%0+%2], %1;" ::"r"(at), "r"(1u), "n"(CT) : "memory");
    }
}
// mass and count of a bin over its copies
__device__ __forceinline__ unsigned long long bin_sums(int bin, uint32_t& count) {
    SampleShared* sh = draw_shared();
    unsigned long long low = 0ull, high = 0ull;
    count = 0u;
#pragma unroll
    for (int i = 0; i < DRAW_LANES; ++i) {                         // (from another copy on in every lane: no two in one bank)
        const int copy_i = (i + bin) % DRAW_LANES;
        low += sh->hist.lo[bin][copy_i];
        high += sh->hist.hi[bin][copy_i];
        count += sh->hist.ct[bin][copy_i];
        if (bin == 255) {
            low += sh->hist.lo[256][copy_i];
            high += sh->hist.hi[256][copy_i];
            count += sh->hist.ct[256][copy_i];
        }
    }
    return low + (high << 20);
}
// A slice of more numbers than the bins' 32-bit sums have room for: segment by segment through them, the sums of all but the last in `tab` and the bins
// empty again for that one; returns its first four.  (2 rows of 486,720 logits with top-p, two segments: 104 us; by radix selects 480.)
__device__ __noinline__ int early_segments(const float* __restrict__ slice, int len, int vec, const DrawBins bins) {
    SampleShared* sh = draw_shared();
    constexpr int STEP = DRAW_SEGMENT / 4;
    const int quads = (len + 3) / 4;
    unsigned long long mass = 0ull;
    uint32_t count = 0u;
    int q0 = 0;
    for (; q0 + STEP < quads; q0 += STEP) {
#pragma unroll 4
        for (int q = q0 + (int)threadIdx.x; q < q0 + STEP; q += DRAW_THREADS) add_to_bins(slice_quad(slice, len, vec, q), bins);
        __syncthreads();
        if (threadIdx.x < 256) {
            uint32_t n;
            mass += bin_sums(threadIdx.x, n);
            count += n;
        }
        __syncthreads();
        for (int i = threadIdx.x; i < (int)(sizeof(sh->hist) / 16); i += DRAW_THREADS) reinterpret_cast<uint4*>(&sh->hist)[i] = make_uint4(0u, 0u, 0u, 0u);
        __syncthreads();
    }
    if (threadIdx.x < 256) {                                       // (read again by the same thread)
        sh->tab.mass[threadIdx.x] = mass;
        sh->tab.ct[threadIdx.x] = count;
    }
    return q0;
}

// Candidates are the elements with key >= floor_key.  In the order (key descending, index ascending) find the
// first element whose cumulative weight exceeds `target`.  Weight is 1 when `by_count`, else the fixed-point
// probability.  Returns the key of that element and how many equal-key elements precede it.
struct SelectResult {
    uint32_t key;
    unsigned long long tie_rank;
};

__device__ __noinline__ SelectResult radix_select(ClusterCtx& c, int begin, int end, float inv_t, float max_scaled, uint32_t floor_key, bool by_count,
                                     unsigned long long target) {
    SampleShared* sh = draw_shared();
    const float* vals = c.vals;                    // (not read anew after every store)
    const int vals_begin = c.vals_begin, copy = (threadIdx.x >> 5) % DRAW_COPIES;
    uint32_t prefix = 0;
    for (int pass = 0; pass < 4; ++pass) {
        const int shift = 24 - 8 * pass;
        __syncthreads();
        for (int i = threadIdx.x; i < DRAW_COPIES * 256; i += DRAW_THREADS) (&sh->whist[0][0])[i] = 0ull;
        __syncthreads();
#pragma unroll 4
        for (int i = begin + (int)threadIdx.x; i < end; i += DRAW_THREADS) {
            const float v = vals[i - vals_begin];
            const uint32_t key = by_count ? order_key(v) : mass_key(v);
            if (key < floor_key) continue;
            if (pass > 0 && (key >> (shift + 8)) != prefix) continue;
            const unsigned long long w = by_count ? 1ull : weight_of(v, inv_t, max_scaled);
            if (w) atomicAdd(&sh->whist[copy][255 - ((key >> shift) & 0xffu)], w);
        }
        __syncthreads();
        const uint32_t b = c.round & 1;
        if (threadIdx.x < 256) {
            unsigned long long sum = 0ull;
#pragma unroll
            for (int w = 0; w < DRAW_COPIES; ++w) sum += sh->whist[w][threadIdx.x];
            sh->pub[b][threadIdx.x] = sum;
        }
        __syncthreads();
        sample_cluster_sync();
        if (threadIdx.x < 256) {
            unsigned long long sum = 0ull, v[SAMPLE_MAX_CLUSTER];
            ld_all_peers_u64(&sh->pub[b][threadIdx.x], c.n_ranks, v);
#pragma unroll
            for (uint32_t r = 0; r < SAMPLE_MAX_CLUSTER; ++r) sum += v[r];
            sh->tot[threadIdx.x] = sum;
        }
        ++c.round;
        pick_bin(target);
        prefix = (prefix << 8) | (255u - sh->chosen);
        target = sh->carry;
    }
    SelectResult r;
    r.key = prefix;
    // all elements with this key have the same logit, hence the same weight
    const unsigned long long w = by_count ? 1ull : weight_of(logit_of_key(prefix), inv_t, max_scaled);
    r.tie_rank = w ? target / w : 0ull;
    return r;
}

__device__ __noinline__ unsigned long long kept_mass(ClusterCtx& c, int begin, int end, float inv_t, float max_scaled, uint32_t floor_key) {
    unsigned long long local = 0;
    const float* vals = c.vals;
    const int vals_begin = c.vals_begin;
#pragma unroll 4
    for (int i = begin + (int)threadIdx.x; i < end; i += DRAW_THREADS) {
        const float v = vals[i - vals_begin];
        if (mass_key(v) >= floor_key) local += weight_of(v, inv_t, max_scaled);
    }
    return cluster_combine(c, local, false);
}

// The bin of a table whose cumulative weight first exceeds `target` (at most the total: beyond it the last element is meant), by
// threads 0 to 255 of those that call it: the thread whose bin it is gets true.
__device__ __forceinline__ bool in_bin(const BinTable* t, int i, bool by_count, unsigned long long target, unsigned long long& carry) {
    const unsigned long long whole = by_count ? (unsigned long long)t->upto_ct[255] : t->upto[255];
    if (target >= whole) target = whole - 1ull;
    const unsigned long long upto = by_count ? (unsigned long long)t->upto_ct[i] : t->upto[i], own = by_count ? (unsigned long long)t->ct[i] : t->mass[i];
    carry = target - (upto - own);
    return target < upto && target >= upto - own;
}

// Bins of two targets, by the whole block, in sh->place: bins of the first level, cut finer where that is at hand.
__device__ __noinline__ void pick_places(bool by_count, unsigned long long target0, unsigned long long target1) {
    SampleShared* sh = draw_shared();
    const int i = threadIdx.x & 255, j = threadIdx.x >> 8;
    const unsigned long long target = j ? target1 : target0;
    static_assert(DRAW_THREADS == 512, "a half of the block per target");
    unsigned long long carry;
    __syncthreads();
    if (in_bin(&sh->tab, i, by_count, target, carry)) sh->place[j] = BinPlace{sh->tab.upto[i] - sh->tab.mass[i], carry, sh->tab.upto[i], i, -1, sh->tab.ct[i]};
    __syncthreads();
    if (!sh->is_fine) return;
    const int bin = sh->place[j].bin;
    const unsigned long long before = sh->place[j].before, rest = sh->place[j].carry;
    int slot = -1;
#pragma unroll
    for (int k = 0; k < DRAW_SLOTS; ++k)
        if (sh->slot_bin[k] == bin) slot = k;
    __syncthreads();
    if (slot >= 0) {
        const BinTable* t = &sh->fine.tab[slot];
        if (in_bin(t, i, by_count, rest, carry)) sh->place[j] = BinPlace{before + t->upto[i] - t->mass[i], carry, before + t->upto[i], bin, i, t->ct[i]};
    }
    __syncthreads();
}

// The same within 256 bins that this CTA filled in sh->cut: place[0] gets the bin as `sub`, its masses after `before`.
__device__ __noinline__ void pick_cut(bool by_count, unsigned long long target, unsigned long long before) {
    SampleShared* sh = draw_shared();
    auto& cut = sh->fine.cut;
    __syncthreads();
    if (threadIdx.x < 256) {
        sh->cut_tab.mass[threadIdx.x] = (unsigned long long)cut.lo[threadIdx.x] + ((unsigned long long)cut.hi[threadIdx.x] << 20);
        sh->cut_tab.ct[threadIdx.x] = cut.ct[threadIdx.x];
    }
    __syncthreads();
    if (threadIdx.x < 32) sum_table(offsetof(SampleShared, cut_tab));
    __syncthreads();
    unsigned long long carry;
    const int i = threadIdx.x & 255;
    if (threadIdx.x < 256 && in_bin(&sh->cut_tab, i, by_count, target, carry))
        sh->place[0] = BinPlace{before + sh->cut_tab.upto[i] - sh->cut_tab.mass[i], carry, before + sh->cut_tab.upto[i], sh->place[0].bin, i, sh->cut_tab.ct[i]};
    __syncthreads();
}

// The search within one bin's entries (sublist) where they are more than DRAW_FEW, by the CTA that holds them: entries in registers, ranges of
// keys cut into 256 bins until all entries left have one key, then the same over their indices.  The result in the found_ fields.
__device__ __noinline__ void search_list(int n, bool by_count, unsigned long long target, unsigned long long before, float inv_t,
                                         float max_scaled) {
    SampleShared* sh = draw_shared();
    constexpr int PER = DRAW_LIST / DRAW_THREADS;
    unsigned long long e[PER];
    bool in[PER];
    uint32_t lo = 0xffffffffu, hi = 0u;
#pragma unroll
    for (int u = 0; u < PER; ++u) {
        const int i = threadIdx.x + u * DRAW_THREADS;
        in[u] = i < n;
        e[u] = in[u] ? sh->fine.sublist[i] : 0ull;
        if (in[u]) {
            lo = min(lo, (uint32_t)(e[u] >> 32));
            hi = max(hi, (uint32_t)(e[u] >> 32));
        }
    }
    auto block_range = [&]() {                     // the smallest and the largest of lo and hi over the block
        __syncthreads();
        if (threadIdx.x == 0) {
            sh->range[0] = 0xffffffffu;
            sh->range[1] = 0u;
        }
        __syncthreads();
        lo = __reduce_min_sync(0xffffffffu, lo);
        hi = __reduce_max_sync(0xffffffffu, hi);
        if ((threadIdx.x & 31) == 0) {
            atomicMin(&sh->range[0], lo);
            atomicMax(&sh->range[1], hi);
        }
        __syncthreads();
        lo = sh->range[0];
        hi = sh->range[1];
    };
    block_range();
    int left = n;
    bool by_index = false;
    unsigned long long w = 0ull, tie = 0ull;
    uint32_t key = 0u;
#pragma unroll 1
    while (true) {                                 // ends: every round leaves a range at most 1/128 as wide, or one key, then one index
        if (lo == hi && by_index) break;
        if (lo == hi) {
            key = lo;
            w = weight_of(logit_of_key(key), inv_t, max_scaled);
            tie = by_count ? target : (w ? target / w : 0ull);
            if (tie >= (unsigned long long)left) tie = (unsigned long long)left - 1ull;
            target = tie;                          // the tie-th smallest index
            by_index = by_count = true;
            lo = 0xffffffffu;
            hi = 0u;
#pragma unroll
            for (int u = 0; u < PER; ++u)
                if (in[u]) {
                    lo = min(lo, (uint32_t)e[u]);
                    hi = max(hi, (uint32_t)e[u]);
                }
            block_range();
            continue;
        }
        const uint32_t old_hi = hi, old_lo = lo;
        const int width = 32 - __clz(hi - lo), s = width > 8 ? width - 8 : 0;
        auto& cut = sh->fine.cut;
        __syncthreads();
        if (threadIdx.x < 256) cut.lo[threadIdx.x] = cut.hi[threadIdx.x] = cut.ct[threadIdx.x] = 0u;
        __syncthreads();
        uint32_t at[PER];
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            at[u] = by_index ? ((uint32_t)e[u] - old_lo) >> s : (old_hi - (uint32_t)(e[u] >> 32)) >> s;
            if (!in[u]) continue;
            const unsigned long long m = by_index ? 0ull : weight_of(logit_of_key((uint32_t)(e[u] >> 32)), inv_t, max_scaled);
            atomicAdd(&cut.lo[at[u]], (uint32_t)m & 0xfffffu);
            atomicAdd(&cut.hi[at[u]], (uint32_t)(m >> 20));
            atomicAdd(&cut.ct[at[u]], 1u);
        }
        pick_cut(by_count, target, before);
        const uint32_t bin = (uint32_t)sh->place[0].sub;
        target = sh->place[0].carry;
        if (!by_index) {
            before = sh->place[0].before;
            left = (int)sh->place[0].count;
        }
        lo = 0xffffffffu;
        hi = 0u;
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            in[u] = in[u] && at[u] == bin;
            if (in[u]) {
                const uint32_t x = by_index ? (uint32_t)e[u] : (uint32_t)(e[u] >> 32);
                lo = min(lo, x);
                hi = max(hi, x);
            }
        }
        block_range();
    }
    if (threadIdx.x == 0) {
        sh->found_key = key;
        sh->found_tie = (uint32_t)tie;
        sh->found_mass = before + w * (unsigned long long)left;
        sh->found_index = lo;
    }
}

__device__ __forceinline__ unsigned long long top_p_need(float P, unsigned long long total) {
    unsigned long long need = (unsigned long long)ceil((double)P * (double)total);
    if (need < 1ull) need = 1ull;
    return need > total ? total : need;
}
__device__ __forceinline__ unsigned long long draw_target(float u, unsigned long long total) {
    const unsigned long long target = (unsigned long long)((double)u * (double)total);
    return target >= total ? total - 1ull : target;
}

// Where the row's searches may end, by the whole block, in sh->want.
__device__ __noinline__ void search_places(int V, int k, float P, float u) {
    SampleShared* sh = draw_shared();
    unsigned long long lo = sh->tab.upto[255], hi = lo;            // what top-k keeps, then what top-p keeps: between these
#pragma unroll 1
    for (int s = 0; s < 3; ++s) {                                  // top-k, top-p, the draw
        if (!(s == 0 ? k > 0 && k < V : s == 1 ? P > 0.0f && P < 1.0f : true)) {
            if (threadIdx.x < 2) sh->want[s][threadIdx.x] = threadIdx.x ? 0.0f : INFINITY;
            continue;
        }
        unsigned long long t0 = (unsigned long long)(k - 1), t1 = t0;
        if (s == 1) {
            lo = top_p_need(P, lo);
            t0 = lo - 1ull;
            t1 = top_p_need(P, hi) - 1ull;
        } else if (s == 2) {
            t0 = draw_target(u, lo);
            t1 = draw_target(u, hi);
        }
        pick_places(s == 0, t0, t1);
        if (threadIdx.x < 2) {
            const int bin = sh->place[threadIdx.x].bin, sub = sh->place[threadIdx.x].sub;
            sh->want[s][threadIdx.x] = (float)(256 * bin + (threadIdx.x ? (sub < 0 ? 256 : sub + 1) : (sub < 0 ? 0 : sub)));
        }
        if (s == 0) {
            lo = max(sh->place[0].before, 1ull);
            hi = max(sh->place[0].upto, 1ull);
        } else if (s == 1) {
            hi = max(min(hi, sh->place[1].upto), lo);
        }
    }
    __syncthreads();
}
__device__ __forceinline__ bool wanted(const SampleShared* sh, float from, float upto) {   // does any of the places lie in [from, upto)
    bool in = false;
#pragma unroll
    for (int s = 0; s < 3; ++s) in |= sh->want[s][0] < upto && sh->want[s][1] > from;
    return in;
}

// One search within the list, by the whole first CTA; the result in the found_ fields.
__device__ __noinline__ void search_bins(const DrawBins bins, bool by_count, unsigned long long target) {
    SampleShared* sh = draw_shared();
    pick_places(by_count, target, target);
    const int n = (int)sh->n_list, bin = sh->place[0].bin;
    if (sh->place[0].sub < 0 && sh->place[0].count > DRAW_FEW) {   // one cut into 256 leaves few
        auto& cut = sh->fine.cut;
        const unsigned long long rest = sh->place[0].carry, before = sh->place[0].before;
        if (threadIdx.x < 256) cut.lo[threadIdx.x] = cut.hi[threadIdx.x] = cut.ct[threadIdx.x] = 0u;
        __syncthreads();
        for (int i = threadIdx.x; i < n; i += DRAW_THREADS) {
            const float v = logit_of_key((uint32_t)(sh->list[i] >> 32));
            const int at = bins.of(v);
            if (at >> 8 != bin) continue;
            const unsigned long long w = weight_below(v, bins.inv_t, bins.max_scaled);
            atomicAdd(&cut.lo[at & 255], (uint32_t)w & 0xfffffu);
            atomicAdd(&cut.hi[at & 255], (uint32_t)(w >> 20));
            atomicAdd(&cut.ct[at & 255], 1u);
        }
        pick_cut(by_count, rest, before);
    }
    const int sub = sh->place[0].sub;
    if (threadIdx.x == 0) sh->few_n = 0u;
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += DRAW_THREADS) {
        const unsigned long long e = sh->list[i];
        const int at = bins.of(logit_of_key((uint32_t)(e >> 32)));
        if (at >> 8 == bin && (sub < 0 || (at & 255) == sub)) sh->fine.sublist[atomicAdd(&sh->few_n, 1u)] = e;
    }
    __syncthreads();
    const int m = (int)sh->few_n;
    if (m > DRAW_FEW) {
        search_list(m, by_count, sh->place[0].carry, sh->place[0].before, bins.inv_t, bins.max_scaled);
        __syncthreads();
        return;
    }
    const unsigned long long e = (int)threadIdx.x < m ? sh->fine.sublist[threadIdx.x] : 0ull;
    const uint32_t key = (uint32_t)(e >> 32), index = (uint32_t)e;
    const unsigned long long w = weight_below(logit_of_key(key), bins.inv_t, bins.max_scaled);
    if ((int)threadIdx.x < m) sh->few_w[threadIdx.x] = w;
    __syncthreads();
    if ((int)threadIdx.x < m) {
        unsigned long long above = 0ull;           // mass, or count, of the entries with larger keys
        unsigned long long above_m = 0ull;
        uint32_t same = 0u, same_before = 0u;
#pragma unroll 4
        for (int i = 0; i < m; ++i) {
            const unsigned long long o = sh->fine.sublist[i];
            const uint32_t okey = (uint32_t)(o >> 32);
            if (okey > key) {
                above_m += sh->few_w[i];
                above += by_count ? 1ull : sh->few_w[i];
            }
            if (okey == key) {
                ++same;
                if ((uint32_t)o < index) ++same_before;
            }
        }
        const unsigned long long one = by_count ? 1ull : w, carry = sh->place[0].carry;
        if (carry >= above && carry < above + one * same && (carry - above) / one == same_before) {
            sh->found_key = key;
            sh->found_index = index;
            sh->found_tie = same_before;
            sh->found_mass = sh->place[0].before + above_m + w * same;
        }
    }
    __syncthreads();
}

// Index of the (rank)-th element, by ascending index, whose key equals `key`; written to out_token by the thread
// that owns it.  False, in every thread of the cluster, if no element has the key.
__device__ __noinline__ bool write_nth_with_key(ClusterCtx& c, int begin, int end, uint32_t key, unsigned long long rank, int32_t* out_token) {
    SampleShared* sh = draw_shared();
    const int len = end - begin;
    const int sub = (len + DRAW_THREADS - 1) / DRAW_THREADS;
    const int lo = begin + min(len, (int)threadIdx.x * sub), hi = begin + min(len, ((int)threadIdx.x + 1) * sub);
    int cnt = 0;
    for (int i = lo; i < hi; ++i) cnt += (order_key(c.vals[i - c.vals_begin]) == key);
    __syncthreads();
    sh->counts[threadIdx.x] = cnt;
    // every CTA publishes how many it holds (cluster_combine would only give the sum: the prefix needs each)
    const unsigned long long mine = warp_sum_u64((unsigned long long)cnt);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) sh->warp_part[warp] = mine;
    __syncthreads();
    const uint32_t b = c.round & 1;
    if (threadIdx.x == 0) {
        unsigned long long v = 0ull;
        for (int w = 0; w < DRAW_WARPS; ++w) v += sh->warp_part[w];
        sh->pub[b][256] = v;
    }
    __syncthreads();
    sample_cluster_sync();
    unsigned long long before = 0ull, total = 0ull, v[SAMPLE_MAX_CLUSTER];
    ld_all_peers_u64(&sh->pub[b][256], c.n_ranks, v);
#pragma unroll
    for (uint32_t r = 0; r < SAMPLE_MAX_CLUSTER; ++r) {
        if (r < c.rank) before += v[r];
        total += v[r];
    }
    ++c.round;
    if (total == 0ull) return false;
    if (rank >= total) rank = total - 1ull;
    const unsigned long long here = sh->pub[b][256];
    if (rank < before || rank >= before + here) return true;      // another CTA's slice holds it
    rank -= before;
    if (threadIdx.x == 0) {
        unsigned long long seen = 0ull;
        int owner = 0;
        for (int t = 0; t < DRAW_THREADS; ++t) {
            if (rank < seen + (unsigned long long)sh->counts[t]) {
                owner = t;
                break;
            }
            seen += (unsigned long long)sh->counts[t];
        }
        sh->chosen = (uint32_t)owner;
        sh->result = (int)(rank - seen);
    }
    __syncthreads();
    if (threadIdx.x == sh->chosen) {
        int seen = 0;
        const int rem = sh->result;
        for (int i = lo; i < hi; ++i)
            if (order_key(c.vals[i - c.vals_begin]) == key) {
                if (seen == rem) {
                    *out_token = i;
                    break;
                }
                ++seen;
            }
    }
    return true;
}

__global__ void __launch_bounds__(DRAW_THREADS, 2)
sample_rows_kernel(const float* __restrict__ logits, int32_t* __restrict__ out, int V,
                   const float* __restrict__ temperature, const int32_t* __restrict__ top_k,
                   const float* __restrict__ top_p, const unsigned long long* __restrict__ seeds,
                   const unsigned long long* __restrict__ counters, int chunk, int vec) {
    extern __shared__ __align__(16) unsigned char sample_smem[];
    ClusterCtx c;
    SampleShared* sh = draw_shared();
    c.rank = blockIdx.x;                                           // the cluster spans x
    c.n_ranks = gridDim.x;
    c.round = 0;
    const int r = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float* row = logits + (size_t)r * V;
    const float T = temperature[r];
    const int k = top_k[r];
    const float P = top_p[r];
    const int begin = min(V, (int)c.rank * chunk), end = min(V, begin + chunk), len = end - begin;
    const int quads = (len + 3) / 4;
    const bool cached = chunk <= DRAW_ROOM;
    auto from_row = [&](int q) { return slice_quad(row + begin, len, vec, q); };
    float4* kept = reinterpret_cast<float4*>(sample_smem + sizeof(SampleShared));
    c.vals = cached ? reinterpret_cast<const float*>(kept) : row;
    c.vals_begin = cached ? begin : 0;
    if (tid == 0) sh->list_n = sh->too_many = 0u;
    // the maximum; NaN takes no part.  Eight loads of 16 bytes a thread are under way together
    float top = NAN;
    bool has_nan = false;
    for (int q0 = tid; q0 < quads; q0 += 8 * DRAW_THREADS) {
        float4 w[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) w[j] = from_row(q0 + j * DRAW_THREADS);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int q = q0 + j * DRAW_THREADS;
            if (q >= quads) break;
            if (cached) kept[q] = w[j];
            top = fmaxf(fmaxf(top, fmaxf(w[j].x, w[j].y)), fmaxf(w[j].z, w[j].w));
            has_nan |= w[j].x != w[j].x || w[j].y != w[j].y || w[j].z != w[j].z || w[j].w != w[j].w;
        }
    }
    for (int i = tid; i < (int)(sizeof(sh->hist) / 16); i += DRAW_THREADS) reinterpret_cast<uint4*>(&sh->hist)[i] = make_uint4(0u, 0u, 0u, 0u);
    {
        const uint32_t best = __reduce_max_sync(0xffffffffu, top != top ? 0u : order_key(top));
        has_nan = __any_sync(0xffffffffu, has_nan);
        if (lane == 0) sh->warp_part[warp] = ((unsigned long long)best << 1) | (has_nan ? 1ull : 0ull);
    }
    __syncthreads();
    if (warp == 0) {
        const unsigned long long p = lane < DRAW_WARPS ? sh->warp_part[lane] : 0ull;
        const uint32_t best = __reduce_max_sync(0xffffffffu, (uint32_t)(p >> 1));
        const bool any = __any_sync(0xffffffffu, (p & 1ull) != 0ull);
        if (lane == 0) sh->pub[0][256] = ((unsigned long long)best << 1) | (any ? 1ull : 0ull);
    }
    sample_cluster_sync();
    uint32_t best = 0u;
    bool nan_in_row = false;
    {
        unsigned long long p[SAMPLE_MAX_CLUSTER];
        ld_all_peers_u64(&sh->pub[0][256], c.n_ranks, p);
#pragma unroll
        for (uint32_t i = 0; i < SAMPLE_MAX_CLUSTER; ++i) {
            best = max(best, (uint32_t)(p[i] >> 1));
            nan_in_row |= (p[i] & 1ull) != 0ull;
        }
    }
    ++c.round;
    // (every path below ends with a cluster barrier: no CTA may exit while a peer still reads its shared memory)
    auto quad = [&](int q) { return cached ? kept[q] : from_row(q); };
    // the lowest index of the maximum; a row without any number gives index 0
    auto write_best = [&]() {
        unsigned long long first = 0ull;
        const float top_logit = logit_of_key(best);
        for (int q = tid; q < quads && first == 0ull && best != 0u; q += DRAW_THREADS) {
            const float4 four = quad(q);
            const float x[4] = {four.x, four.y, four.z, four.w};
            if (!(fmaxf(fmaxf(x[0], x[1]), fmaxf(x[2], x[3])) >= top_logit)) continue;
#pragma unroll
            for (int j = 3; j >= 0; --j)
                if (__float_as_uint(x[j]) == __float_as_uint(top_logit) && 4 * q + j < len) first = (uint32_t)~(uint32_t)(begin + 4 * q + j);
        }
        first = cluster_combine(c, first, true);
        if (c.rank == 0 && tid == 0) out[r] = first ? (int)~(uint32_t)first : 0;
        sample_cluster_sync();
    };
    if (T <= 0.0f || k == 1 || best == 0u) {
        write_best();
        return;
    }
    const float max_logit = logit_of_key(best);
    const float inv_t = 1.0f / T;
    const float max_scaled = max_logit * inv_t;
    const uint64_t bits = mix64(seeds[r], counters[r]);
    const float u = (float)(bits >> 40) * (1.0f / 16777216.0f);  // 24 bits → [0,1)
    // Below 2^21 max_scaled is off by 1/16 at most, so that no weight exceeds FIXED_ONE e^(1/16) and the sums of the bins have room; NaN and
    // infinities are not below it.
    const bool plain = !nan_in_row && fabsf(max_scaled) < 2097152.0f && isfinite(inv_t) && inv_t > 0.0f;
    if (plain) {
        const DrawBins bins{inv_t, max_scaled, inv_t * 0.03125f, max_scaled * 0.03125f};
        // slices of more than 60,800 numbers: all segments but the last, their sums in `tab`
        const int q_first = len > DRAW_SEGMENT ? early_segments(row + begin, len, vec, bins) : 0;
#pragma unroll 2
        for (int q = q_first + tid; q < quads; q += DRAW_THREADS) add_to_bins(quad(q), bins);
        __syncthreads();
        if (tid < 256) {
            uint32_t count;
            unsigned long long mass = bin_sums(tid, count);
            if (q_first > 0) {
                mass += sh->tab.mass[tid];
                count += sh->tab.ct[tid];
            }
            sh->pub[1][tid] = mass;
            sh->pub_ct[tid] = tid == 255 ? count - (uint32_t)(4 * quads - len) : count;
        }
        sample_cluster_sync();
        if (tid < 256) {
            unsigned long long p[SAMPLE_MAX_CLUSTER], mass = 0ull;
            ld_all_peers_u64(&sh->pub[1][tid], c.n_ranks, p);
#pragma unroll
            for (uint32_t i = 0; i < SAMPLE_MAX_CLUSTER; ++i) mass += p[i];
            sh->tab.mass[tid] = mass;
        } else {
            sh->tab.ct[tid - 256] = sum_all_peers_u32(&sh->pub_ct[tid - 256], c.n_ranks);
        }
        if (tid < DRAW_SLOTS) sh->slot_bin[tid] = -1;
        if (tid == 0) sh->is_fine = 0u;
        __syncthreads();
        if (warp == 0) sum_table(offsetof(SampleShared, tab));
        __syncthreads();
        bool fits = false, listed = false;
        int slots = 0;
        uint32_t n_near = 0u;
        // every number of the bins that hold places, as of the first round: from the warp's list, or from the slice if that has overflowed
        auto each_near = [&](auto use) {
            if (listed) {
                for (uint32_t i = lane; i < n_near; i += 32) {
                    const int at = sh->near[warp][i];
                    use(c.vals[at + begin - c.vals_begin], at);
                }
            } else {
                for (int i = tid; i < len; i += DRAW_THREADS) {
                    const float y = c.vals[i + begin - c.vals_begin];
                    if (sh->marked[min(bins.of(y) >> 8, 255)]) use(y, i);
                }
            }
        };
        auto& f = sh->fine;
        for (int round = 0;; ++round) {
            if (tid == 0) sh->n_list = 0u;
            search_places(V, k, P, u);
            // how many numbers lie in these places; which bins they are
            if (warp < 8) {
                const bool in = wanted(sh, 256.0f * (float)tid, 256.0f * (float)(tid + 1));
                bool cut = false;
#pragma unroll
                for (int i = 0; i < DRAW_SLOTS; ++i) cut |= sh->slot_bin[i] == tid;
                const uint32_t all = __ballot_sync(0xffffffffu, in), n = __reduce_add_sync(0xffffffffu, in && !cut ? sh->tab.ct[tid] : 0u);
                const uint32_t open = __ballot_sync(0xffffffffu, in && !cut);
                if (lane == 0) {
                    sh->mask[warp] = all;
                    if (n) atomicAdd(&sh->n_list, n);
                    sh->warp_part[warp] = open;
                }
            }
            for (int i = tid; i < 256 * slots; i += DRAW_THREADS) {
                const float at = (float)(256 * sh->slot_bin[i >> 8] + (i & 255));
                const uint32_t n = f.tab[i >> 8].ct[i & 255];
                if (n && wanted(sh, at, at + 1.0f)) atomicAdd(&sh->n_list, n);
            }
            __syncthreads();
            if (round == 0) {
                // the numbers of these bins, from the slice; a quarter of a warp's words has none nearer than the last of the bins
                if (tid < 256) sh->marked[tid] = (unsigned char)((sh->mask[warp] >> lane) & 1u);
                if (tid == 256) sh->marked[256] = (unsigned char)(sh->mask[7] >> 31);
                int last = 0;
#pragma unroll
                for (int w = 0; w < 8; ++w)
                    if (sh->mask[w]) last = 32 * w + 31 - __clz(sh->mask[w]);
                const float nearer = last == 255 ? INFINITY : (float)(last + 1) / 256.0f;
                const uint32_t mark = (uint32_t)__cvta_generic_to_shared(&sh->marked[0]) - 0x4b000000u;
                __syncthreads();
#pragma unroll 1
                for (int q0 = warp * 32; q0 < quads && len <= DRAW_SEGMENT; q0 += DRAW_THREADS) {      // (the lists hold places in 16 bits)
                    const int q = q0 + lane;
                    const float4 four = q < quads ? quad(q) : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
                    const float x[4] = {four.x, four.y, four.z, four.w};
                    if (!__any_sync(0xffffffffu, bins.below(fmaxf(fmaxf(x[0], x[1]), fmaxf(x[2], x[3]))) < nearer)) continue;
                    uint32_t m[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        asm volatile("ld.shared.u8 %0, [%1];" : "=r"(m[j]) : "r"(bins.first_bits(x[j]) + mark) : "memory");
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const bool in = m[j] != 0u && 4 * q + j < len;
                        const uint32_t all = __ballot_sync(0xffffffffu, in);
                        const uint32_t at = n_near + (uint32_t)__popc(all & ((1u << lane) - 1u));
                        if (in && at < DRAW_NEAR) sh->near[warp][at] = (unsigned short)(4 * q + j);
                        n_near += (uint32_t)__popc(all);
                    }
                }
                listed = !__syncthreads_or(n_near > DRAW_NEAR) && len <= DRAW_SEGMENT;
            }
            fits = sh->n_list <= DRAW_LIST;
            if (fits || round == 2) break;
            int n_bins = 0, before = 0;
            bool open = false;
            const int only = k > 0 && k < V ? (int)sh->want[0][0] >> 8 : -1;   // of too many bins, top-k's own: the others are fewer once its place is known
#pragma unroll
            for (int w = 0; w < 8; ++w) {
                const uint32_t m = sh->mask[w];
                if (w < warp) before += __popc(m);
                if (w == warp) before += __popc(m & ((1u << lane) - 1u));
                n_bins += __popc(m);
                open |= sh->warp_part[w] != 0ull;
            }
            if (!open || (n_bins > DRAW_SLOTS && (only < 0 || round > 0))) break;     // (nearly) equal logits, or masses of many bins in doubt
            const bool all_bins = n_bins <= DRAW_SLOTS;
            slots = all_bins ? n_bins : 1;
            __syncthreads();
            if (tid < DRAW_SLOTS) sh->slot_bin[tid] = -1;
            if (tid < 256) sh->slot_of[tid] = 0;
            __syncthreads();
            if (warp < 8 && (all_bins ? ((sh->mask[warp] >> lane) & 1u) != 0u : tid == only)) {
                const int slot = all_bins ? before : 0;
                sh->slot_bin[slot] = tid;
                sh->slot_of[tid] = (unsigned char)(slot + 1);
            }
            for (int i = tid; i < 256 * slots; i += DRAW_THREADS) f.lo[i] = f.hi[i] = f.ct[i] = 0u;
            __syncthreads();
            each_near([&](float y, int) {
                const int at = bins.of(y), slot = (int)sh->slot_of[at >> 8] - 1, i = 256 * slot + (at & 255);
                if (slot < 0) return;
                const Halves w = weight_halves(y, inv_t, max_scaled);
                atomicAdd(&f.lo[i], w.low);
                if (w.high) atomicAdd(&f.hi[i], w.high);
                atomicAdd(&f.ct[i], 1u);
            });
            __syncthreads();
            for (int i = tid; i < 256 * slots; i += DRAW_THREADS) f.pub[i] = (unsigned long long)f.lo[i] + ((unsigned long long)f.hi[i] << 20);
            sample_cluster_sync();
            for (int i = tid; i < 256 * slots; i += DRAW_THREADS) {
                unsigned long long p[SAMPLE_MAX_CLUSTER], mass = 0ull;
                ld_all_peers_u64(&f.pub[i], c.n_ranks, p);
#pragma unroll
                for (uint32_t j = 0; j < SAMPLE_MAX_CLUSTER; ++j) mass += p[j];
                const uint32_t count = sum_all_peers_u32(&f.ct[i], c.n_ranks);
                f.tab[i >> 8].mass[i & 255] = mass;
                f.tab[i >> 8].ct[i & 255] = count;
                if (count > DRAW_LO_MAX) sh->too_many = 1u;        // (nearly) equal logits: 32 bits may not have held the low halves
            }
            if (tid == 0) sh->is_fine = 1u;
            __syncthreads();
            if (warp < slots) sum_table((uint32_t)(offsetof(SampleShared, fine.tab) + warp * sizeof(BinTable)));
            __syncthreads();
            if (sh->too_many != 0u) break;
            sample_cluster_sync();                                 // the peers have read this CTA's sums
        }
        if (fits) {
            const float a0 = sh->want[0][0], a1 = sh->want[0][1], b0 = sh->want[1][0], b1 = sh->want[1][1], c0 = sh->want[2][0], c1 = sh->want[2][1];
            unsigned long long* own = f.own;                       // (beside the warps' lists, which take the place of the cluster's)
            each_near([&](float y, int i) {
                const float place = bins.place(y);
                if (!((place >= a0 && place < a1) || (place >= b0 && place < b1) || (place >= c0 && place < c1))) return;
                const uint32_t at = atomicAdd(&sh->list_n, 1u);
                if (at < DRAW_LIST) own[at] = ((unsigned long long)order_key(y) << 32) | (uint32_t)(begin + i);
            });
            sample_cluster_sync();
            if (c.rank != 0) {
                sample_cluster_sync();                             // until the first CTA has the lists
                return;
            }
            uint32_t held[SAMPLE_MAX_CLUSTER];
#pragma unroll
            for (uint32_t i = 0; i < SAMPLE_MAX_CLUSTER; ++i) {
                held[i] = 0u;
                if (i < c.n_ranks) asm volatile("ld.shared::cluster.u32 %0, [%1];\n" : "=r"(held[i]) : "r"(peer_address(&sh->list_n, i)) : "memory");
            }
            unsigned long long e[SAMPLE_MAX_CLUSTER];
#pragma unroll
            for (uint32_t i = 0; i < SAMPLE_MAX_CLUSTER; ++i)
                if (tid < (int)held[i]) e[i] = ld_peer_u64(&f.own[tid], i);
            uint32_t at = 0u;
#pragma unroll
            for (uint32_t i = 0; i < SAMPLE_MAX_CLUSTER; ++i) {    // (n_list of them in all, at most DRAW_LIST)
                if (tid < (int)held[i]) sh->list[at + tid] = e[i];
                for (uint32_t j = tid + DRAW_THREADS; j < held[i]; j += DRAW_THREADS) sh->list[at + j] = ld_peer_u64(&f.own[j], i);
                at += held[i];
            }
            asm volatile("barrier.cluster.arrive.release;\n" ::: "memory");
            // the three searches, one after the other
            uint32_t floor_key = 0u;
            unsigned long long total = sh->tab.upto[255];
            if (k > 0 && k < V) {
                search_bins(bins, true, (unsigned long long)(k - 1));
                floor_key = sh->found_key;
                total = sh->found_mass;
            }
            if (P > 0.0f && P < 1.0f) {                            // the smallest prefix whose cumulative share reaches P
                search_bins(bins, false, top_p_need(P, total) - 1ull);
                if (sh->found_key > floor_key) {
                    floor_key = sh->found_key;
                    total = sh->found_mass;
                }
            }
            search_bins(bins, false, draw_target(u, total));
            if (tid == 0) out[r] = (int)sh->found_index;
            asm volatile("barrier.cluster.wait.acquire;\n" ::: "memory");
            return;
        }
        sample_cluster_sync();                                     // the radix select's sums take the place of what peers may be reading
    }
    // every other row: radix selects over the slice
    // top-k: everything at or above the k-th largest logit stays
    uint32_t floor_key = 0;
    if (k > 0 && k < V) floor_key = radix_select(c, begin, end, inv_t, max_scaled, 0u, true, (unsigned long long)(k - 1)).key;
    unsigned long long total = kept_mass(c, begin, end, inv_t, max_scaled, floor_key);
    if (total == 0ull) {  // numerical underflow: the reference falls back to the best candidate
        write_best();
        return;
    }
    // top-p: the smallest prefix whose cumulative share reaches P
    if (P > 0.0f && P < 1.0f) {
        const SelectResult s = radix_select(c, begin, end, inv_t, max_scaled, floor_key, false, top_p_need(P, total) - 1ull);
        if (s.key > floor_key) floor_key = s.key;
        total = kept_mass(c, begin, end, inv_t, max_scaled, floor_key);
    }
    const SelectResult s = radix_select(c, begin, end, inv_t, max_scaled, floor_key, false, draw_target(u, total));
    if (!write_nth_with_key(c, begin, end, s.key, s.tie_rank, &out[r])) {
        write_best();
        return;
    }
    sample_cluster_sync();
}

MM_EXPORT int mm_sample_rows(const void* logits, void* out, int R, int V, const void* temperature, const void* top_k,
                             const void* top_p, const void* seeds, const void* counters, void* stream) {
    MM_REQUIRE(R >= 0 && R <= 65535 && V > 0, "sample: bad sizes");
    if (R == 0) return MM_OK;
    // A row is shared by a cluster of CTAs (a power of two: other sizes place badly): enough that their shared memory holds a copy of it, more
    // while the launch leaves SMs idle and a slice keeps 4096 numbers.
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    int ranks = 1;
    while (ranks < SAMPLE_MAX_CLUSTER && ((V + ranks - 1) / ranks > DRAW_ROOM || (V / (ranks * 2) >= 4096 && (long long)R * ranks * 2 <= sms))) ranks *= 2;
    const int vec = V % 4 == 0 && reinterpret_cast<uintptr_t>(logits) % 16 == 0;
    const int chunk = ((V + ranks - 1) / ranks + 3) / 4 * 4;
    const size_t smem = sizeof(SampleShared) + (chunk <= DRAW_ROOM ? (size_t)chunk * sizeof(float) : 0);
    if (!mm_allow_smem<sample_rows_kernel>(sizeof(SampleShared) + DRAW_ROOM * sizeof(float))) {
        mm_set_last_error("sample: cannot reserve shared memory");
        return MM_ERR_LAUNCH;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ranks, R);
    cfg.blockDim = dim3(DRAW_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ranks;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ranks > 1 ? 1 : 0;
    cudaLaunchKernelEx(&cfg, sample_rows_kernel, (const float*)logits, (int32_t*)out, V, (const float*)temperature,
                       (const int32_t*)top_k, (const float*)top_p, (const unsigned long long*)seeds,
                       (const unsigned long long*)counters, chunk, vec);
    MM_CHECK_LAUNCH();
    return MM_OK;
}

// ---- soft-cap and penalties, in place on the logits ---------------------------
// recent: int32 [R, W] (entries < 0 are padding).  For each distinct recent token t with
// count c: l = l > 0 ? l / rep : l * rep; l -= freq * c; l -= pres.
__global__ void penalties_kernel(float* __restrict__ logits, int V, const int32_t* __restrict__ recent, int W,
                                 const float* __restrict__ rep, const float* __restrict__ freq,
                                 const float* __restrict__ pres, const float* __restrict__ softcap) {
    const int r = blockIdx.x;
    float* row = logits + (size_t)r * V;
    const float cap = softcap ? softcap[r] : 0.0f;
    if (cap > 0.0f) {
        const float inv = 1.0f / cap;
        for (int i = threadIdx.x; i < V; i += blockDim.x) row[i] = cap * tanhf(row[i] * inv);
        __syncthreads();
    }
    if (recent == nullptr || W <= 0) return;
    const float rp = rep[r], fp = freq[r], pp = pres[r];
    if (rp == 1.0f && fp == 0.0f && pp == 0.0f) return;
    const int32_t* win = recent + (size_t)r * W;
    for (int i = threadIdx.x; i < W; i += blockDim.x) {
        const int t = win[i];
        if (t < 0 || t >= V) continue;
        int count = 0;
        bool first = true;
        for (int j = 0; j < W; ++j) {
            if (win[j] == t) {
                ++count;
                if (j < i) first = false;
            }
        }
        if (!first) continue;
        float l = row[t];
        if (rp != 1.0f) l = (l > 0.0f) ? (l / rp) : (l * rp);
        if (fp != 0.0f) l -= fp * (float)count;
        if (pp != 0.0f) l -= pp;
        row[t] = l;
    }
}

MM_EXPORT int mm_apply_penalties(void* logits, int R, int V, const void* recent, int W, const void* rep,
                                 const void* freq, const void* pres, const void* softcap, void* stream) {
    MM_REQUIRE(R >= 0 && V > 0 && W >= 0, "penalties: bad sizes");
    if (R == 0) return MM_OK;
    penalties_kernel<<<R, 256, 0, (cudaStream_t)stream>>>((float*)logits, V, (const int32_t*)recent, W, (const float*)rep,
                                                          (const float*)freq, (const float*)pres, (const float*)softcap);
    MM_CHECK_LAUNCH();
    return MM_OK;
}

// recent: int32 [R, W] rings of the last widths[r] tokens of each row (entries beyond the width, or not yet filled,
// are -1); lengths[r] counts the row's tokens so far.  Puts tokens[r] at lengths[r] % widths[r] and advances the count:
// the window of a captured decode step follows the sequence without the host.
__global__ void window_push_kernel(int32_t* __restrict__ recent, int W, const int32_t* __restrict__ widths,
                                   long long* __restrict__ lengths, const int32_t* __restrict__ tokens, int R) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= R) return;
    const int w = widths[r] < W ? widths[r] : W;
    if (w > 0) recent[(size_t)r * W + (int)(lengths[r] % w)] = tokens[r];
    lengths[r] += 1;
}

MM_EXPORT int mm_window_push(void* recent, int R, int W, const void* widths, void* lengths, const void* tokens, void* stream) {
    MM_REQUIRE(R >= 0 && W >= 1, "window_push: bad sizes");
    if (R == 0) return MM_OK;
    window_push_kernel<<<(R + 127) / 128, 128, 0, (cudaStream_t)stream>>>((int32_t*)recent, W, (const int32_t*)widths,
                                                                         (long long*)lengths, (const int32_t*)tokens, R);
    MM_CHECK_LAUNCH();
    return MM_OK;
}

// After a decode step: every request's position moves on by one, its draw counter too (null: no counters), and the
// sampled tokens become the next step's inputs (null: the caller feeds them).
__global__ void advance_step_kernel(int32_t* __restrict__ positions, long long* __restrict__ counters, int32_t* __restrict__ next_ids,
                                    const int32_t* __restrict__ tokens, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    positions[i] += 1;
    if (counters != nullptr) counters[i] += 1;
    if (next_ids != nullptr) next_ids[i] = tokens[i];
}

MM_EXPORT int mm_advance_step(void* positions, void* counters, void* next_ids, const void* tokens, int n, void* stream) {
    MM_REQUIRE(n >= 0 && positions != nullptr && (next_ids == nullptr || tokens != nullptr), "advance_step: bad arguments");
    if (n == 0) return MM_OK;
    advance_step_kernel<<<(n + 127) / 128, 128, 0, (cudaStream_t)stream>>>((int32_t*)positions, (long long*)counters, (int32_t*)next_ids,
                                                                          (const int32_t*)tokens, n);
    MM_CHECK_LAUNCH();
    return MM_OK;
}

// uniform number of (seed, counter), exported so the host-side plain sampler draws the same stream
MM_EXPORT float mm_uniform_from(unsigned long long seed, unsigned long long counter) {
    return (float)(mix64(seed, counter) >> 40) * (1.0f / 16777216.0f);
}
