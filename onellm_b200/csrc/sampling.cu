// Top-K selection and top-K sampling for sm_100a.
//
// Top-K generalises the reference's two-round block top-K with K fixed at 2
// (src/kernels/beamsearch_topK.cu:20-119, struct topK in src/kernels/beamsearch_topK.h:3-33)
// to 1 <= K <= 64 with a defined order for ties (lower column first).  Sampling restates
// SamplingKernel (src/kernels/topK_sampling.cu:6-41) with the same cuRAND call sequence.
//
// One thread block per row, over an order-preserving integer image of the logits (NaN lowest).  Rows of up to
// 32768 logits (topk_reg_kernel) are read once, 32 keys per thread in registers: the K-th largest of
// the maxima of groups of keys bounds the K-th largest key from below, the few keys that reach it are gathered and ranked
// against each other; rows with long runs of equal keys fall back to a bisection over all keys.  Neither step
// uses a histogram: logits share their leading bits, and a 256-bin histogram in shared memory serialises on a
// handful of bins.  Longer rows (topk_kernel) are a radix select, 8 bits per pass, re-reading the logits from L2.
#include <curand_kernel.h>
#include <math.h>

#include <algorithm>
#include <type_traits>

#include "common.cuh"

namespace onellm {

constexpr int kTopkThreads = 1024;
constexpr int kMaxK = 64;

__device__ __forceinline__ uint32_t float_key(float f)
{
    if (f != f) return 0u;  // NaN sorts below everything
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ float key_float(uint32_t k)
{
    const uint32_t u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
    return __uint_as_float(u);
}

template <typename T>
__device__ __forceinline__ float load_logit(const T* p, int i);
template <>
__device__ __forceinline__ float load_logit<float>(const float* p, int i) { return p[i]; }
template <>
__device__ __forceinline__ float load_logit<__half>(const __half* p, int i) { return __half2float(p[i]); }

template <typename T>
__global__ void __launch_bounds__(kTopkThreads)
topk_kernel(const T* __restrict__ logits, int vocab, int K, float* __restrict__ out_val, int* __restrict__ out_id,
            int global_ids)
{
    pdl_launch_dependents();
    pdl_wait();
    const int row = blockIdx.x;
    const T* x = logits + (size_t)row * vocab;
    __shared__ int hist[256];
    __shared__ uint32_t s_prefix;
    __shared__ int s_need;            // how many still to take among keys matching the prefix
    __shared__ int s_count;           // gather cursor
    __shared__ int warp_tot[kTopkThreads / 32];
    __shared__ uint32_t cand_key[kMaxK];
    __shared__ int cand_id[kMaxK];

    if (threadIdx.x == 0) {
        s_prefix = 0u;
        s_need = K;
        s_count = 0;
    }
    __syncthreads();

    // 1. K-th largest key, 8 bits at a time from the top
    for (int pass = 0; pass < 4; pass++) {
        const int shift = 24 - 8 * pass;
        const uint32_t mask = pass == 0 ? 0u : (0xffffffffu << (shift + 8));
        for (int i = threadIdx.x; i < 256; i += kTopkThreads) hist[i] = 0;
        __syncthreads();
        const uint32_t prefix = s_prefix;
        for (int i = threadIdx.x; i < vocab; i += kTopkThreads) {
            const uint32_t k = float_key(load_logit<T>(x, i));
            if ((k & mask) == prefix) atomicAdd(&hist[(k >> shift) & 255u], 1);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            int need = s_need, b = 255;
            for (; b > 0; b--) {
                if (hist[b] >= need) break;
                need -= hist[b];
            }
            s_prefix = prefix | ((uint32_t)b << shift);
            s_need = need;  // ties still to take once all 32 bits are fixed
        }
        __syncthreads();
    }
    const uint32_t kth = s_prefix;
    const int need_ties = s_need;

    // 2. gather: everything above the K-th key (any order), then the lowest-indexed ties
    for (int i = threadIdx.x; i < vocab; i += kTopkThreads) {
        const uint32_t k = float_key(load_logit<T>(x, i));
        if (k > kth) {
            const int pos = atomicAdd(&s_count, 1);
            cand_key[pos] = k;
            cand_id[pos] = i;
        }
    }
    __syncthreads();
    const int n_above = s_count;  // == K - need_ties
    {
        // contiguous slices per thread so that an exclusive scan gives ranks in column order
        const int per = (vocab + kTopkThreads - 1) / kTopkThreads;
        const int c0 = threadIdx.x * per, c1 = min(c0 + per, vocab);
        int mine = 0;
        for (int i = c0; i < c1; i++) mine += (float_key(load_logit<T>(x, i)) == kth);
        int incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if ((threadIdx.x & 31) >= o) incl += v;
        }
        if ((threadIdx.x & 31) == 31) warp_tot[threadIdx.x >> 5] = incl;
        __syncthreads();
        if (threadIdx.x < 32) {
            int v = threadIdx.x < kTopkThreads / 32 ? warp_tot[threadIdx.x] : 0;
            int inc = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, inc, o);
                if (threadIdx.x >= o) inc += u;
            }
            if (threadIdx.x < kTopkThreads / 32) warp_tot[threadIdx.x] = inc - v;  // exclusive
        }
        __syncthreads();
        int rank = warp_tot[threadIdx.x >> 5] + incl - mine;
        for (int i = c0; i < c1 && rank < need_ties; i++) {
            if (float_key(load_logit<T>(x, i)) == kth) {
                cand_key[n_above + rank] = kth;
                cand_id[n_above + rank] = i;
                rank++;
            }
        }
    }
    __syncthreads();

    // 3. rank sort: larger key first, lower column first among equals
    if (threadIdx.x < K) {
        const uint32_t k = cand_key[threadIdx.x];
        const int id = cand_id[threadIdx.x];
        int r = 0;
        for (int j = 0; j < K; j++) r += (cand_key[j] > k) || (cand_key[j] == k && cand_id[j] < id);
        const float v = key_float(k);
        out_val[(size_t)row * K + r] = (k == 0u) ? -INFINITY : v;
        out_id[(size_t)row * K + r] = global_ids ? row * vocab + id : id;
    }
}


template <typename T>
__device__ __forceinline__ uint32_t logit_key(T v);
template <>
__device__ __forceinline__ uint32_t logit_key<float>(float v) { return float_key(v); }
template <>
__device__ __forceinline__ uint32_t logit_key<__half>(__half v)
{
    // 16-bit image in the upper half of the key: same order as the float image, two radix passes
    const uint32_t u = __half_as_ushort(v);
    if ((u & 0x7fffu) > 0x7c00u) return 0u;  // NaN
    return ((u & 0x8000u) ? (~u & 0xffffu) : (u | 0x8000u)) << 16;
}
template <typename T>
__device__ __forceinline__ float key_value(uint32_t k);
template <>
__device__ __forceinline__ float key_value<float>(uint32_t k) { return key_float(k); }
template <>
__device__ __forceinline__ float key_value<__half>(uint32_t k)
{
    const uint32_t k16 = k >> 16;
    const uint32_t u = (k16 & 0x8000u) ? (k16 & 0x7fffu) : (~k16 & 0xffffu);
    return __half2float(__ushort_as_half((unsigned short)u));
}

// The draw of (step, row) is curand_init(step, row, 0) + curand_uniform, as src/kernels/topK_sampling.cu:29-30 of the
// reference takes it.  For row > 0 nearly all of its time is the skip-ahead to sub-sequence `row`: a linear map
// (over GF(2)) of the 160 xorshift bits of the XORWOW state, which cuRAND applies bit by bit in one thread, 10-15 us
// per set bit of the row index.  The map depends on the row only, so a caller that draws for the same rows at
// every step can have it tabulated once (build_skip_table: the image of each of the 160 unit vectors under
// skipahead_sequence(row), 3200 bytes per row, and the change of the additive counter `d`); the draw is then
// curand_init(step, 0, 0), which skips nothing, and an XOR of the columns the state's set bits select, five bits per
// lane.  The table is checked against the direct form when it is built and not used if a single draw differs.
constexpr int kSkipBits = 160, kSkipWords = 5;
constexpr int kSkipRowWords = kSkipBits * kSkipWords + 1;  // a row's columns, then its counter change

__global__ void skip_table_kernel(uint32_t* __restrict__ tab)
{
    const int b = blockIdx.x, i = threadIdx.x;  // one row per block, one state bit per thread
    curandStateXORWOW_t s;
    s.d = 0u;
    for (int w = 0; w < kSkipWords; w++) s.v[w] = 0u;
    s.boxmuller_flag = 0;
    s.boxmuller_flag_double = 0;
    s.boxmuller_extra = 0.f;
    s.boxmuller_extra_double = 0.0;
    s.v[i >> 5] = 1u << (i & 31);
    skipahead_sequence((unsigned long long)b, &s);
    uint32_t* row = tab + (size_t)b * kSkipRowWords;
    for (int w = 0; w < kSkipWords; w++) row[i * kSkipWords + w] = s.v[w];
    if (i == 0) row[kSkipBits * kSkipWords] = s.d;
}

// Whole warp; the result is valid in lane 0.
__device__ __forceinline__ float draw_with_table(int seed, int b, const uint32_t* __restrict__ tab)
{
    const uint32_t* row = tab + (size_t)b * kSkipRowWords;
    const int lane = threadIdx.x & 31;
    curandStateXORWOW_t s;
    uint32_t v[kSkipWords] = {0u, 0u, 0u, 0u, 0u};
    if (lane == 0) {
        curand_init((unsigned long long)seed, 0ULL, 0ULL, &s);
#pragma unroll
        for (int w = 0; w < kSkipWords; w++) v[w] = s.v[w];
    }
#pragma unroll
    for (int w = 0; w < kSkipWords; w++) v[w] = __shfl_sync(0xffffffffu, v[w], 0);
    uint32_t acc[kSkipWords] = {0u, 0u, 0u, 0u, 0u};
#pragma unroll
    for (int q = 0; q < kSkipBits / 32; q++) {
        const int bit = q * 32 + lane;  // word q, bit `lane`
        if ((v[q] >> lane) & 1u) {
            const uint32_t* col = row + bit * kSkipWords;
#pragma unroll
            for (int w = 0; w < kSkipWords; w++) acc[w] ^= col[w];
        }
    }
#pragma unroll
    for (int w = 0; w < kSkipWords; w++) acc[w] = __reduce_xor_sync(0xffffffffu, acc[w]);
    float u = 0.f;
    if (lane == 0) {
#pragma unroll
        for (int w = 0; w < kSkipWords; w++) s.v[w] = acc[w];
        s.d += row[kSkipBits * kSkipWords];
        u = curand_uniform(&s);
    }
    return u;
}

__global__ void skip_table_check_kernel(const uint32_t* __restrict__ tab, int* __restrict__ mismatches)
{
    const int b = blockIdx.x;
    const int seeds[6] = {0, 1, 2, 515, 12345, 0x7fffffff};
    for (int i = 0; i < 6; i++) {
        const float fast = draw_with_table(seeds[i], b, tab);
        if (threadIdx.x == 0) {
            curandState_t state;
            curand_init((unsigned long long)seeds[i], (unsigned long long)b, 0ULL, &state);
            if (curand_uniform(&state) != fast) atomicAdd(mismatches, 1);
        }
    }
}

// What a draw of step and row decides and where that goes
struct SampleTo {
    float temperature;
    const int* step;  // device
    int vocab, end_id, literal_walk;
    int *id, *id2, *host_id;  // id2 and host_id may be null
    int* seqlen;              // with finished, or both null
    unsigned char* finished;
    float* u;  // may be null
    const uint32_t* skip_tab;
};

// Whole warp; the result is valid in lane 0.
__device__ __noinline__ float draw_of(int seed, int b, const uint32_t* tab)
{
    float u = 0.f;
    if (tab) {
        u = draw_with_table(seed, b, tab);
    } else if ((threadIdx.x & 31) == 0) {
        curandState_t state;
        curand_init((unsigned long long)seed, (unsigned long long)b, 0ULL, &state);
        u = curand_uniform(&state);
    }
    return u;
}

// One thread; weight(i): the i-th candidate's
template <typename W>
__device__ __forceinline__ int walk(int K, float u, int literal_walk, W weight)
{
    float sum = 0.f;
    for (int i = 0; i < K; i++) sum += weight(i);
    float thr = u * sum;
    for (int i = 0; i < K; i++) {
        thr -= literal_walk ? 1.0f : weight(i);
        if (thr < 0.f) return i;
    }
    return K - 1;
}

__device__ __forceinline__ void sampled(const SampleTo& to, int b, int id, float u)
{
    to.id[b] = id;
    if (to.u) to.u[b] = u;
    if (to.id2) to.id2[b] = id;
    if (to.host_id) to.host_id[b] = id;
    if (to.seqlen && to.finished) {
        to.seqlen[b] = to.finished[b] ? to.seqlen[b] : to.seqlen[b] + 1;
        to.finished[b] = (id == to.end_id) ? 1 : 0;
    }
}

constexpr int kTopkPer = 32;  // keys per thread held in registers
constexpr int kTopkCand = 512;  // gathered keys the short way ranks; >= kMaxK

// SAMPLE: and the sampling from them.  What bounds it is the chain of one block's barriers behind the logits, most of a step's LM head being
// hidden: the draw is taken before the logits are there, the weights of the candidates are computed side by side.  A launch less:
// with the loads below, prompts and 16 steps of float logits (K = 1) 5755 -> 5650 and 5590 -> 5480 us.
template <typename T, bool SAMPLE>
__global__ void __launch_bounds__(kTopkThreads)
topk_reg_kernel(const T* __restrict__ logits, int vocab, int K, float* __restrict__ out_val, int* __restrict__ out_id,
                int global_ids, const SampleTo to)
{
    constexpr int VEC = 16 / sizeof(T);
    pdl_launch_dependents();
    const int row = blockIdx.x, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __shared__ int s_count;
    __shared__ int warp_tot[kTopkThreads / 32];
    __shared__ uint32_t cand_key[kTopkCand];
    __shared__ int cand_id[kTopkCand];
    __shared__ float best_val[SAMPLE ? kMaxK : 1];
    __shared__ int best_id[SAMPLE ? kMaxK : 1];
    // The step counter was written by work that completed long before: it is advanced by the first kernel of a step, and the layer
    // projections between it and this kernel release their dependents only after passing their own griddepcontrol.wait.
    float u = 0.f;
    if (SAMPLE && wid == 0) u = draw_of(*to.step, row, to.skip_tab);
    pdl_wait();
    const T* x = logits + (size_t)row * vocab;

    // A warp reads 512 bytes side by side.  32 columns side by side in a thread make a load of floats one of 32 cache lines: 32000 columns,
    // K = 1, us, then | now: float 10.3 | 4.8, half 5.7 | 5.7.
    auto col_of = [](int j) { return ((j / VEC) * kTopkThreads + (int)threadIdx.x) * VEC + j % VEC; };
    uint32_t key[kTopkPer];
    if (vocab % VEC == 0 && (reinterpret_cast<uintptr_t>(x) & 15u) == 0) {
#pragma unroll
        for (int j = 0; j < kTopkPer; j += VEC) {
            uint4 raw = make_uint4(~0u, ~0u, ~0u, ~0u);  // NaN: key 0
            if (col_of(j) < vocab) raw = *reinterpret_cast<const uint4*>(x + col_of(j));
            const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
            for (int q = 0; q < VEC; q++) key[j + q] = logit_key<T>(e[q]);
        }
    } else {
#pragma unroll
        for (int j = 0; j < kTopkPer; j++) key[j] = col_of(j) < vocab ? logit_key<T>(x[col_of(j)]) : 0u;
    }
    if (threadIdx.x == 0) s_count = 0;
    __syncthreads();

    constexpr int kLowBit = sizeof(T) == 2 ? 16 : 0;  // fp16 keys live in the upper half
    __shared__ int bit_tot[2][kTopkThreads / 32];
    __shared__ __align__(16) uint32_t maxima[kTopkThreads];
    __shared__ uint32_t s_low;
    int it = 0;
    bool done = false;

    auto put = [&](int r, uint32_t k, int id) {
        const float v = (k == 0u) ? -INFINITY : key_value<T>(k);
        out_val[(size_t)row * K + r] = v;
        out_id[(size_t)row * K + r] = global_ids ? row * vocab + id : id;
        if constexpr (SAMPLE) best_val[r] = v, best_id[r] = id;
    };

    // 0. The short way, which nearly every row of logits takes.  The K-th largest of the maxima of groups of keys is a lower bound of the
    // K-th largest key (K groups hold a key that large), and for logits hardly more than K keys reach it: of G groups of columns in any
    // order the keys of G ln(G / (G - K)) threads.  The groups are, up to K = 16, the 32 warps, whose maxima every warp ranks (22 threads
    // at K = 16); above, eight lanes each, 63 threads at K = 50, and one warp bisects their 128 maxima.  The keys that reach the bound
    // are gathered (a few dozen shared-memory atomics) and ranked against each other, larger key first, lower column first among
    // equals: rank r < K is output slot r.  Where many more do (the large logits side by side in few groups) or the row is
    // short, the bound comes from the maxima of all threads; rows with many equal keys, where that gathers too many as well, take the
    // bisection over all keys below.  8 x 32000, us, with the bound of all threads and
    // a barrier a bit | now: K = 50 half 10.1 | 9.8, float 17.3 | 10.0; sorted rows 29.5 | 31.1, 48.5 | 21.1; three values 28.2 | 27.6, 47.1 | 40.1.
    {
        uint32_t mk = 0u;  // padding and NaN have key 0
#pragma unroll
        for (int j = 0; j < kTopkPer; j++) mk = max(mk, key[j]);
        auto filled = [&](int lanes) { return min(kTopkThreads, (vocab + VEC - 1) / VEC) / lanes; };  // whole groups of so many lanes
        auto bisect = [&](auto n) {  // one warp: the K-th largest of 128 n maxima
            const uint32_t at = (uint32_t)__cvta_generic_to_shared(maxima + 4 * lane);
            uint32_t lo = 0u;
#pragma unroll 1
            for (int bit = 31; bit >= kLowBit; bit--) {
                const uint32_t t = lo | (1u << bit);
                int c = 0, d = 0;
#pragma unroll
                for (int i = 0; i < decltype(n)::value; i++) {
                    uint4 m;  // again for every bit: there are no registers to keep them in
                    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(m.x), "=r"(m.y), "=r"(m.z), "=r"(m.w) : "r"(at + i * 512) : "memory");
                    c += (m.x >= t) + (m.y >= t);
                    d += (m.z >= t) + (m.w >= t);
                }
                if ((int)__reduce_add_sync(0xffffffffu, c + d) >= K) lo = t;
            }
            return lo;
        };
        for (int way = 2 * K <= filled(32) ? 0 : 2 * K <= filled(8) ? 1 : 2; way < 3 && !done; way = way < 2 ? 2 : 3) {
            uint32_t low = 0u;
            if (way == 0) {
                const uint32_t wm = __reduce_max_sync(0xffffffffu, mk);
                if (lane == 0) maxima[wid] = wm;
                __syncthreads();
                const uint32_t v = maxima[lane];
                int r = 0;
#pragma unroll
                for (int j = 0; j < 32; j++) {
                    const uint32_t u = __shfl_sync(0xffffffffu, v, j);
                    r += u > v || (u == v && j < lane);
                }
                low = __shfl_sync(0xffffffffu, v, __ffs(__ballot_sync(0xffffffffu, r == K - 1)) - 1);
            } else {
                uint32_t gm = mk;
                if (way == 1) {
                    gm = max(gm, __shfl_xor_sync(0xffffffffu, gm, 1));
                    gm = max(gm, __shfl_xor_sync(0xffffffffu, gm, 2));
                    gm = max(gm, __shfl_xor_sync(0xffffffffu, gm, 4));
                }
                if (way == 2) maxima[threadIdx.x] = gm;
                else if ((lane & 7) == 0) maxima[threadIdx.x / 8] = gm;
                __syncthreads();
                if (wid == 0) {
                    low = way == 1 ? bisect(std::integral_constant<int, 1>{}) : bisect(std::integral_constant<int, kTopkThreads / 128>{});
                    if (lane == 0) s_low = low;
                }
                __syncthreads();
                low = s_low;
            }
            // twice what columns in any order lead to, and more
            if (way < 2 && __syncthreads_count(mk >= low) > (way == 0 ? 64 : 160)) continue;
            low = max(low, 1u);  // 0: NaN, or no column
            if (mk >= low) {
#pragma unroll
                for (int j = 0; j < kTopkPer; j++) {
                    if (key[j] >= low) {
                        const int pos = atomicAdd(&s_count, 1);
                        if (pos < kTopkCand) {
                            cand_key[pos] = key[j];
                            cand_id[pos] = col_of(j);
                        }
                    }
                }
            }
            __syncthreads();
            const int n_c = s_count;  // >= K where K threads hold a key above 0
            if (n_c >= K && n_c <= kTopkCand) {
                if ((int)threadIdx.x < n_c) {
                    const uint32_t k = cand_key[threadIdx.x];
                    const int id = cand_id[threadIdx.x];
                    int r = 0;
                    for (int j = 0; j < n_c; j++) r += (cand_key[j] > k) || (cand_key[j] == k && cand_id[j] < id);
                    if (r < K) put(r, k, id);
                }
                done = true;
                break;
            }
            __syncthreads();  // everyone has read s_count
            if (threadIdx.x == 0) s_count = 0;
            __syncthreads();
        }
    }

    if (!done) {
        // 1. K-th largest key by bisection on its bits, from the top: the largest t with at least K keys >= t.  Every thread
        // counts its 32 keys in registers, a warp adds up with one reduction, the 32 warp sums meet in shared memory (two
        // buffers in turn: one block barrier per bit) and every thread takes the same decision, so nothing is broadcast
        // and no shared-memory atomic is used (a 256-bin histogram of logits has a handful of hot bins: the radix form
        // of this step spent most of its 39 us waiting for them).
        auto block_count = [&](auto pred) {
            int c = 0;
#pragma unroll
            for (int j = 0; j < kTopkPer; j++) c += pred(key[j]) ? 1 : 0;
            c = __reduce_add_sync(0xffffffffu, c);
            int* tot = bit_tot[it++ & 1];
            if (lane == 0) tot[wid] = c;
            __syncthreads();
            return (int)__reduce_add_sync(0xffffffffu, tot[lane]);
        };
        uint32_t kth = 0u;
#pragma unroll 1
        for (int bit = 31; bit >= kLowBit; bit--) {
            const uint32_t t = kth | (1u << bit);
            if (block_count([t](uint32_t k) { return k >= t; }) >= K) kth = t;
        }
        const bool all_ties = block_count([kth](uint32_t k) { return k >= kth; }) == K;  // kth == 0: the places without a column count too

        // 2. gather: everything above the K-th key (any order), and its ties where all of them count
#pragma unroll
        for (int j = 0; j < kTopkPer; j++) {
            if (key[j] > kth || (all_ties && key[j] == kth)) {
                const int pos = atomicAdd(&s_count, 1);
                cand_key[pos] = key[j];
                cand_id[pos] = col_of(j);
            }
        }
        __syncthreads();
        // else the lowest-indexed ties: a thread's VEC columns, then the threads, then the groups of columns follow each other
        int n = s_count;
#pragma unroll
        for (int g = 0; g < kTopkPer / VEC; g++) {
            if (n < K) {
                int ties = 0;
#pragma unroll
                for (int q = 0; q < VEC; q++) ties += key[g * VEC + q] == kth && col_of(g * VEC + q) < vocab;
                int incl = ties;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += v;
                }
                if (lane == 31) warp_tot[wid] = incl;
                __syncthreads();
                const int before = __reduce_add_sync(0xffffffffu, lane < wid ? warp_tot[lane] : 0);
                const int all = __reduce_add_sync(0xffffffffu, warp_tot[lane]);
                int at = n + before + incl - ties;
#pragma unroll
                for (int q = 0; q < VEC; q++) {
                    if (key[g * VEC + q] == kth && col_of(g * VEC + q) < vocab) {
                        if (at < K) {
                            cand_key[at] = kth;
                            cand_id[at] = col_of(g * VEC + q);
                        }
                        at++;
                    }
                }
                n += all;
                __syncthreads();
            }
        }

        // 3. rank sort: larger key first, lower column first among equals
        if (threadIdx.x < K) {
            const uint32_t k = cand_key[threadIdx.x];
            const int id = cand_id[threadIdx.x];
            int r = 0;
            for (int j = 0; j < K; j++) r += (cand_key[j] > k) || (cand_key[j] == k && cand_id[j] < id);
            put(r, k, id);
        }
    }

    if constexpr (SAMPLE) {
        __syncthreads();
        if (wid > 0) return;
        float* weight = reinterpret_cast<float*>(cand_key);
        for (int i = lane; i < K; i += 32) weight[i] = expf((best_val[i] - best_val[0]) / to.temperature);
        __syncwarp();
        if (lane == 0) sampled(to, row, best_id[walk(K, u, to.literal_walk, [&](int i) { return weight[i]; })] % to.vocab, u);
    }
}

__global__ void sample_kernel(const int* __restrict__ topk_id, const float* __restrict__ topk_val, int K, int rng_step, const SampleTo to, int early_seed)
{
    pdl_launch_dependents();
    const int b = blockIdx.x;
    // The draw depends on (step, row) only, and seeding the generator (a sequence skip-ahead) is by far
    // the longest part of this kernel.  early_seed: do it before waiting for the candidates; the caller
    // vouches that *to.step was written by work that completed long before (see topk_reg_kernel).
    float u = 0.f;
    auto draw = [&]() { u = draw_of(to.step ? *to.step : rng_step, b, to.skip_tab); };
    if (early_seed) draw();
    pdl_wait();
    if (!early_seed) draw();
    if (threadIdx.x != 0) return;
    const float* v = topk_val + (size_t)b * K;
    const float v0 = v[0];
    const int pick = walk(K, u, to.literal_walk, [&](int i) { return expf((v[i] - v0) / to.temperature); });
    sampled(to, b, topk_id[(size_t)b * K + pick] % to.vocab, u);
}

// Rows that topk_reg_kernel takes
template <typename T, bool SAMPLE>
static int topk_launch(const void* logits, int rows, int vocab, int K, float* out_val, int* out_id, int global_ids, const SampleTo& to, cudaStream_t st)
{
    ONELLM_CUDA(launch_pdl(topk_reg_kernel<T, SAMPLE>, dim3(rows), dim3(kTopkThreads), 0, st, (const T*)logits, vocab, K, out_val, out_id, global_ids, to));
    ONELLM_CHECK_LAUNCH();
    return ONELLM_OK;
}

}  // namespace onellm

using namespace onellm;

extern "C" int onellm_topk(int dtype, const void* logits, int rows, int vocab, int K, float* out_val, int* out_id,
                           int global_ids, void* stream)
{
    ONELLM_REQUIRE(logits && out_val && out_id, ONELLM_ERR_ARG, "topk: null pointer");
    ONELLM_REQUIRE(rows >= 0 && vocab > 0, ONELLM_ERR_ARG, "topk: bad size");
    ONELLM_REQUIRE(K >= 1 && K <= kMaxK && K <= vocab, ONELLM_ERR_UNSUPPORTED, "topk: K=%d outside [1, %d]", K,
                   kMaxK);
    if (rows == 0) return ONELLM_OK;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    ONELLM_REQUIRE(dtype == ONELLM_F16 || dtype == ONELLM_F32, ONELLM_ERR_UNSUPPORTED, "topk: dtype %d", dtype);
    if (vocab <= kTopkPer * kTopkThreads)
        return dtype == ONELLM_F16 ? topk_launch<__half, false>(logits, rows, vocab, K, out_val, out_id, global_ids, SampleTo{}, st)
                                   : topk_launch<float, false>(logits, rows, vocab, K, out_val, out_id, global_ids, SampleTo{}, st);
    if (dtype == ONELLM_F16)
        ONELLM_CUDA(launch_pdl(topk_kernel<__half>, dim3(rows), dim3(kTopkThreads), 0, st, (const __half*)logits, vocab, K, out_val, out_id, global_ids));
    else
        ONELLM_CUDA(launch_pdl(topk_kernel<float>, dim3(rows), dim3(kTopkThreads), 0, st, (const float*)logits, vocab, K, out_val, out_id, global_ids));
    ONELLM_CHECK_LAUNCH();
    return ONELLM_OK;
}

namespace onellm {
static int sample_launch(const int* topk_id, const float* topk_val, int B, int K, int rng_step, const SampleTo& to, bool early_seed, cudaStream_t st)
{
    ONELLM_REQUIRE(topk_id && topk_val && to.id, ONELLM_ERR_ARG, "topk_sample: null pointer");
    ONELLM_REQUIRE(B >= 0 && K >= 1 && to.vocab > 0 && to.temperature > 0.f, ONELLM_ERR_ARG,
                   "topk_sample: bad size or temperature");
    ONELLM_REQUIRE((to.seqlen == nullptr) == (to.finished == nullptr), ONELLM_ERR_ARG,
                   "topk_sample: seqlen and finished must be given together");
    if (B == 0) return ONELLM_OK;
    ONELLM_CUDA(launch_pdl(sample_kernel, dim3(B), dim3(32), 0, st, topk_id, topk_val, K, rng_step, to, early_seed ? 1 : 0));
    return ONELLM_OK;
}

// The model driver's top-K and sampling of B rows of logits, in one launch where a row fits a block's registers.  output_id2 gets a
// second copy of the sampled ids (the next step's input buffer), host_id one in mapped host memory.
int sample_logits(int dtype, const void* logits, int B, int vocab, int K, float* topk_val, int* topk_id, float temperature, const int* step, int end_id,
                  int literal_walk, int* output_id, int* seqlen, unsigned char* finished, float* u_out, int* output_id2, int* host_id,
                  const uint32_t* skip_table, cudaStream_t st)
{
    const SampleTo to = {temperature, step, vocab, end_id, literal_walk, output_id, output_id2, host_id, seqlen, finished, u_out, skip_table};
    if (vocab > kTopkPer * kTopkThreads || K < 1 || K > std::min(kMaxK, vocab) || (dtype != ONELLM_F16 && dtype != ONELLM_F32)) {
        const int rc = onellm_topk(dtype, logits, B, vocab, K, topk_val, topk_id, 0, (void*)st);
        return rc != ONELLM_OK ? rc : sample_launch(topk_id, topk_val, B, K, 0, to, /*early_seed=*/true, st);
    }
    return dtype == ONELLM_F16 ? topk_launch<__half, true>(logits, B, vocab, K, topk_val, topk_id, 0, to, st)
                               : topk_launch<float, true>(logits, B, vocab, K, topk_val, topk_id, 0, to, st);
}

// Words a skip table for `rows` rows takes.
size_t skip_table_words(int rows) { return (size_t)rows * kSkipRowWords; }

// Fills `table` (device memory, skip_table_words(rows) words) for rows 0..rows-1 and checks it against the direct
// draw; waits for the stream.  *usable = 0 when a draw differed (the caller then passes no table).  A table built
// for `rows` rows serves launches of up to that many rows.
int build_skip_table(uint32_t* table, int rows, int* usable, cudaStream_t st)
{
    ONELLM_REQUIRE(table && usable && rows > 0, ONELLM_ERR_ARG, "skip table: bad argument");
    int* d_bad = nullptr;
    ONELLM_CUDA(cudaMalloc(&d_bad, sizeof(int)));
    cudaError_t e = cudaMemsetAsync(d_bad, 0, sizeof(int), st);
    if (e == cudaSuccess) {
        skip_table_kernel<<<rows, kSkipBits, 0, st>>>(table);
        skip_table_check_kernel<<<rows, 32, 0, st>>>(table, d_bad);
        e = cudaGetLastError();
    }
    int bad = 1;
    if (e == cudaSuccess) e = cudaMemcpyAsync(&bad, d_bad, sizeof(int), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(d_bad);
    ONELLM_CUDA(e);
    *usable = bad == 0 ? 1 : 0;
    return ONELLM_OK;
}
}  // namespace onellm

extern "C" int onellm_topk_sample(const int* topk_id, const float* topk_val, int B, int K, float temperature,
                                  int rng_step, const int* rng_step_dev, int vocab_size, int end_id,
                                  int literal_walk, int* output_id, int* seqlen, unsigned char* finished,
                                  float* u_out, void* stream)
{
    const SampleTo to = {temperature, rng_step_dev, vocab_size, end_id, literal_walk, output_id, nullptr, nullptr, seqlen, finished, u_out, nullptr};
    return sample_launch(topk_id, topk_val, B, K, rng_step, to, /*early_seed=*/false, reinterpret_cast<cudaStream_t>(stream));
}
