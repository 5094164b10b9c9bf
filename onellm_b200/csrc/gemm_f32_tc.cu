// float32 projections of more than 64 tokens on the tensor cores, with the precision of float.
//
// Replaces the cuBLAS SGEMM behind launchLinearGemm (src/kernels/qkv_linear.cu:8-65 of the reference) for context passes of
// float32 callers.  A float is the sum of three bf16 values, each the nearest to what the ones before it leave (the method of Henry,
// Tang and Heinecke, "Leveraging the bfloat16 Artificial Intelligence Datatype For Higher-Precision Computations", 2019):
// x = x0 + x1 + x2, |x1| <= 2^-8 |x|, |x2| <= 2^-17 |x|.  Of the nine products of two such sums eight are computed; x2 w2, below
// 2^-34 of x w, is not.
//
// A block computes y^T: 128 columns of W are the rows of the MMA, the tokens (at most 192) its columns, so that a token count
// that is no multiple of 128 costs no padding.
//   W      lane = column: a thread splits 8 rows of its column and stores the pieces to tensor memory, where the MMA takes its A
//          operand from: no transposition.
//   x      8 threads split the 32 values of a token's stage; the pieces go to shared memory in the 128-byte swizzled form
//          ([x0 | x1] in one tile of 128-byte rows, [x2 | unused] in a second one).
//          Both come as floats by TMA, three stages ahead.
//   sums   the tensor cores add into a float with truncation, so an accumulator is not kept for long: every stage of 32 rows
//          starts a new one, the seven small products go in before x0 w0, and the warps then add it to their
//          registers, rounding to nearest.  Two accumulators, two buffers of each operand: the warps add stage s - 1 and
//          convert stage s + 1 while the MMAs of stage s run.
// K is split over the blocks of a cluster where the tiles alone would not fill the GPU; the partial sums meet in distributed
// shared memory in rank order.
// What bounds it: a stage of 176 tokens takes about 2100 cycles, 1400 of them its MMAs; the warps split its floats, add an accumulator
// and wait for both one after the other.  Sixteen warps instead of eight shorten that chain, with half of the rows, columns and
// registers each: 352 tokens of the 7B shapes, us (with eight | the 64 x 64 tiled kernel): QKV 266 (276 | 2209), o_proj 90 (91 | 911),
// gate or up 245 (250 | 2202), down 217 (219 | 2569), 131 to 146 TFLOP/s of float32; a layer 1355 (1390).  Error against 64 bits, normal
// operands, 1.1e-7 (chain 1.1e-6; K = 11008: 1.5e-7, 1.8e-6), a layer 6.9e-7 instead of 2.8e-6.
// What the pieces do not hold: a value that is not finite, or whose first piece rounds to infinity, makes its remainders NaN and so
// every result it enters; one below 2^-110 loses its last bits.  Blocks whose results that touches (see `stands`) compute them
// again by plain multiply-adds, at the rate of the tiled kernel; the results are that kernel's to the bit.
#include <cooperative_groups.h>

#include <algorithm>
#include <mutex>

#include "gemm_f32.h"
#include "tc_common.cuh"

namespace cg = cooperative_groups;

namespace onellm {

constexpr int kFtCols = 128;                    // columns of W per block
constexpr int kFtTok = 192;                     // most tokens per block
constexpr int kFtK = 32;                        // rows of W per stage
constexpr int kFtWarps = 16;                    // warps that convert and add, four to 32 columns of W
constexpr int kFtParts = kFtWarps / 4;
constexpr int kFtThreads = kFtWarps * 32 + 32;  // and one that issues loads and MMAs
constexpr int kFtTile = kFtTok * 128;           // bytes: a 128-byte row per token
constexpr int kFtPiecesBytes = 4 * kFtTile;     // two stages of two tiles; the partial sums of the cluster afterwards
constexpr int kFtDepth = 3;                     // stages of floats on their way
constexpr int kFtRawW = kFtK * kFtCols * 4, kFtRaw = kFtRawW + kFtTok * kFtK * 4;
constexpr int kFtSmem = kFtPiecesBytes + kFtDepth * kFtRaw;
constexpr int kFtGroup = kFtTok / kFtParts / 3; // accumulator columns read at a time
// The third piece of a float below 2^-110 falls among the subnormal bf16 values and loses up to 2^-133, on either side of a product: a
// result of K products beside the largest operand then counts from 2^26 times K * 2^-132 of it.  Below kFtLeast the products of
// the pieces themselves leave the range of float.
constexpr float kFtLost = 0x1p-106f, kFtLeast = 0x1p-80f;
constexpr unsigned kGaveUp = 0xffffffffu;  // above the bits of every float that is not NaN
constexpr uint32_t kFtPieces = 2 * kFtTok;      // tensor memory: two accumulators, then two stages of 3 pieces x 16 columns
static_assert(kFtGroup == 16 && kFtPieces + 2 * 48 <= 512 && kFtTok * kFtCols * 4 <= kFtPiecesBytes, "layout");

__device__ __forceinline__ void finish_f32(const GemmF32& a, int m, int n, float v)
{
    const size_t at = (size_t)m * a.ldy + n;
    if (a.resid) v = fmaf(v, a.scale, a.resid[at]);
    if (a.gate >= 0) v = gate_pair<true>(a.y[at], v, a.gate, a.limit);
    a.y[at] = v;
}

// This thread's share of the largest operand of a block, 16 bytes at a time (K, and N of W [K,N], are multiples of 4)
template <bool NK>
__device__ __noinline__ float largest(const GemmF32& a, int m0, int rows, int n0, int k_begin, int k_end)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n_end = min(n0 + kFtCols, a.N);
    float top = 0.f;
    auto take = [&](const float* p) {
        const float4 v = *reinterpret_cast<const float4*>(p);
        top = fmaxf(fmaxf(top, fmaxf(fabsf(v.x), fabsf(v.y))), fmaxf(fabsf(v.z), fabsf(v.w)));
    };
    auto rows_of = [&](const float* p, int begin, int end, long ld) {
        for (int r = begin + warp; r < end; r += kFtThreads / 32)
#pragma unroll 8
            for (int k = k_begin + 4 * lane; k < k_end; k += 128) take(p + (size_t)r * ld + k);
    };
    rows_of(a.x, m0, m0 + rows, a.ldx);
    if constexpr (NK) {
        rows_of(a.W, n0, n_end, a.ldw);
    } else if (n0 + 4 * lane < n_end) {
#pragma unroll 8
        for (int k = k_begin + warp; k < k_end; k += kFtThreads / 32) take(a.W + (size_t)k * a.ldw + n0 + 4 * lane);
    }
    return top;
}

// The outputs of `rows` tokens from m0 on and the block's columns by multiply-adds in the order of k, as sgemm_kernel adds them: 64 tokens
// at a time, 4 x 8 outputs a thread, the operands of the next 32 k on their way meanwhile.  All threads of the block call it (the last
// warp for the barriers); buf: kFtPlainBytes of shared memory.
constexpr int kFtPlainK = 32, kFtPlainTok = 64;
constexpr int kFtPlainBytes = kFtPlainK * (kFtPlainTok + 4 + kFtCols + 4) * 4;
static_assert(kFtPlainBytes <= kFtDepth * kFtRaw, "in place of the floats");
template <bool NK>
__device__ __noinline__ void plain_tile(const GemmF32& a, float* buf, int m0, int rows, int n0)
{
    float(*xs)[kFtPlainTok + 4] = reinterpret_cast<float(*)[kFtPlainTok + 4]>(buf);
    float(*ws)[kFtCols + 4] = reinterpret_cast<float(*)[kFtCols + 4]>(buf + kFtPlainK * (kFtPlainTok + 4));
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const bool works = tid < 256;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int t0 = 0; t0 < rows; t0 += kFtPlainTok) {
        // four values of k of a token, or of a column; W [K,N]: four columns.  K, and N there, are multiples of 4.
        float4 xv[2], wv[4];
        auto fetch = [&](int k0) {
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const int e = tid + 256 * i, t = t0 + (e >> 3), k = k0 + (e & 7) * 4;
                xv[i] = works && t < rows && k < a.K ? *reinterpret_cast<const float4*>(a.x + (size_t)(m0 + t) * a.ldx + k) : zero;
            }
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int e = tid + 256 * i, n = n0 + (NK ? e >> 3 : (e & 31) * 4), k = k0 + (NK ? (e & 7) * 4 : e >> 5);
                wv[i] = works && n < a.N && k < a.K ? *reinterpret_cast<const float4*>(a.W + (NK ? (size_t)n * a.ldw + k : (size_t)k * a.ldw + n)) : zero;
            }
        };
        float acc[4][8] = {};
        fetch(0);
        for (int k0 = 0; k0 < a.K; k0 += kFtPlainK) {
            __syncthreads();
            if (works) {
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const int e = tid + 256 * i, t = e >> 3, k = (e & 7) * 4;
                    xs[k][t] = xv[i].x, xs[k + 1][t] = xv[i].y, xs[k + 2][t] = xv[i].z, xs[k + 3][t] = xv[i].w;
                }
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int e = tid + 256 * i, c = e >> 3, k = (e & 7) * 4;
                    if constexpr (NK) ws[k][c] = wv[i].x, ws[k + 1][c] = wv[i].y, ws[k + 2][c] = wv[i].z, ws[k + 3][c] = wv[i].w;
                    else *reinterpret_cast<float4*>(&ws[e >> 5][(e & 31) * 4]) = wv[i];
                }
            }
            __syncthreads();
            if (k0 + kFtPlainK < a.K) fetch(k0 + kFtPlainK);
            const int steps = works ? min(kFtPlainK, a.K - k0) : 0;
#pragma unroll 4
            for (int kk = 0; kk < steps; kk++) {
                float x[4], w[8];
                *reinterpret_cast<float4*>(x) = *reinterpret_cast<const float4*>(&xs[kk][ty * 4]);
                *reinterpret_cast<float4*>(w) = *reinterpret_cast<const float4*>(&ws[kk][tx * 4]);
                *reinterpret_cast<float4*>(w + 4) = *reinterpret_cast<const float4*>(&ws[kk][64 + tx * 4]);
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int j = 0; j < 8; j++) acc[i][j] = fmaf(x[i], w[j], acc[i][j]);
            }
        }
        if (works) {
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const int t = t0 + ty * 4 + i, n = n0 + (j >> 2) * 64 + tx * 4 + (j & 3);
                    if (t < rows && n < a.N) finish_f32(a, m0 + t, n, acc[i][j]);
                }
        }
    }
}

// grid (ceil(N / 128), K split, ceil(M / nt)), cluster (1, K split, 1); nt: tokens per block, a multiple of 16; every block has a stage
template <bool NK>
__global__ void __launch_bounds__(kFtThreads, 1)
gemm_f32_tc_kernel(const GemmF32 a, const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, int nt, int stages_per_block)
{
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bars[4 + kFtDepth];  // pieces of a stage are there (2), its products are done (2), its floats are there
    __shared__ uint32_t tmem_slot;
    __shared__ unsigned s_top;  // of the cluster: 0, or the largest operand of ranks that have one which is not the sum of its pieces
                                // (bits of a float), or kGaveUp
    cg::cluster_group cluster = cg::this_cluster();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n0 = blockIdx.x * kFtCols, m0 = blockIdx.z * nt, m_rows = min(nt, a.M - m0);
    const int k_begin = blockIdx.y * stages_per_block * kFtK, k_end = min(k_begin + stages_per_block * kFtK, a.K);
    const int n_stages = (k_end - k_begin + kFtK - 1) / kFtK;
    const uint32_t full0 = smem_u32(bars), done0 = smem_u32(bars + 2), raw0 = smem_u32(bars + 4);
    bool ok = (smem_u32(smem_raw) & 1023u) == 0;  // the swizzle works on address bits
    if (!ok && tid == 0) atomicExch(&g_tc_timeout_flag, 1);
    if (tid == 0) {
        for (int s = 0; s < 2; s++) {
            mbar_init(full0 + 8 * s, kFtWarps);
            mbar_init(done0 + 8 * s, 1);
        }
        for (int s = 0; s < kFtDepth; s++) mbar_init(raw0 + 8 * s, 1);
        s_top = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    if (gridDim.y > 1) cluster_arrive();
    pdl_wait();

    const int part = warp >> 2, np = nt / kFtParts;  // a warp adds the accumulator columns [part * np, part * np + np) of its 32 lanes
    float acc[3 * kFtGroup];
#pragma unroll
    for (int i = 0; i < 3 * kFtGroup; i++) acc[i] = 0.f;

    int loaded = 0, issued = 0;  // stages, of the warp that issues
    bool lossy = false;          // pieces of this thread's operands do not add up to them
    if (warp == kFtWarps) {
        // Issues the loads of the floats and the MMAs (the whole warp runs this; one elected lane issues)
        const uint64_t desc = umma_desc(smem_u32(smem_raw), 16, 1024);
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(nt >> 3) << 17) | ((uint32_t)(kFtCols >> 4) << 24);
        const uint32_t raw = smem_u32(smem_raw) + kFtPiecesBytes;
        const bool leader = elect_one();
        auto fetch = [&](int s, int slot) {
            if (!leader || s >= n_stages) return;
            const int k0 = k_begin + s * kFtK;
            const uint32_t bar = raw0 + 8 * slot, dst = raw + (uint32_t)(slot * kFtRaw);
            mbar_expect_tx(bar, (uint32_t)(kFtRawW + nt * kFtK * 4));
            if constexpr (NK) tma_load_2d(dst, &map_w, k0, n0, bar);
            else tma_load_2d(dst, &map_w, n0, k0, bar);
            tma_load_2d(dst + kFtRawW, &map_x, k0, m0, bar);
        };
        if (ok)
            for (int s = 0; s < kFtDepth; s++) fetch(s, s);
        if (ok) loaded = min(n_stages, kFtDepth);
        int slot = 0;
        for (int s = 0; s < n_stages && ok; s++) {
            ok = mbar_wait_warp(full0 + 8 * (s & 1), (uint32_t)(s >> 1) & 1u);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            fetch(s + kFtDepth, slot);  // every warp has split the floats of this stage
            loaded = min(n_stages, s + 1 + kFtDepth);
            slot = slot + 1 == kFtDepth ? 0 : slot + 1;
            if (leader) {
                const uint32_t d = tmem + (uint32_t)((s & 1) * kFtTok), wp = tmem + kFtPieces + (uint32_t)((s & 1) * 48);
                const uint64_t xd = desc + (uint64_t)((s & 1) * (2 * kFtTile >> 4));
                constexpr int kW[8] = {1, 2, 2, 0, 1, 1, 0, 0}, kX[8] = {2, 1, 0, 2, 1, 0, 1, 0};  // pieces of the products, small ones first
#pragma unroll
                for (int i = 0; i < 8; i++)
#pragma unroll
                    for (int kk = 0; kk < 2; kk++)
                        umma_f16_tmem_a(d, wp + kW[i] * 16 + kk * 8, xd + (uint64_t)(((kX[i] >> 1) * kFtTile + (kX[i] & 1) * 64 + kk * 32) >> 4), idesc,
                                        i + kk > 0 ? 1u : 0u);
                umma_commit(done0 + 8 * (s & 1));
            }
            issued++;
            __syncwarp();
        }
    } else {
        const uint32_t t_lane = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        const int col = (warp & 3) * 32 + lane;
        // x: rows r and r + 4 of a group of 8 side by side, so that a warp's stores fill all banks
        const int quad = tid & 7, row0 = (warp * 4 & ~7) + ((tid >> 3) & 1) * 4 + ((tid >> 4) & 1) + (warp & 1) * 2;
        const uint32_t x_at = (uint32_t)row0 * 128 + (((quad >> 1) ^ (row0 & 7)) << 4) + (quad & 1) * 8;  // + 64 rows: + 8192
        auto add = [&](int s) {
            if (!mbar_wait_warp(done0 + 8 * (s & 1), (uint32_t)(s >> 1) & 1u)) return false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int g = 0; g < 3; g++) {
                if (g * kFtGroup < np) {
                    uint32_t v[kFtGroup];
                    tmem_ld16(t_lane + (uint32_t)((s & 1) * kFtTok + part * np + g * kFtGroup), v);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int i = 0; i < kFtGroup; i++) acc[g * kFtGroup + i] += __uint_as_float(v[i]);
                }
            }
            return true;
        };
        uint32_t rest = 0u;
        int slot = 0;
        uint32_t phase = 0;
        for (int s = 0; s < n_stages && ok; s++) {
            ok = mbar_wait_warp(raw0 + 8 * slot, phase);
            if (!ok) break;
            const unsigned char* raw = smem_raw + kFtPiecesBytes + slot * kFtRaw;
            // the buffers of this stage were last read by the MMAs of stage s - 2, whose accumulator has been added
            uint32_t p0[4], p1[4], p2[4];
            if constexpr (NK) {  // [128 columns][32 k], 128-byte swizzled
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const float4 v = *reinterpret_cast<const float4*>(raw + col * 128 + (((part * 2 + i) ^ (col & 7)) << 4));
                    split_pair(v.x, v.y, p0[2 * i], p1[2 * i], p2[2 * i], rest);
                    split_pair(v.z, v.w, p0[2 * i + 1], p1[2 * i + 1], p2[2 * i + 1], rest);
                }
            } else {  // [32 k][128 columns]
                const float* wr = reinterpret_cast<const float*>(raw) + part * 8 * kFtCols + col;
#pragma unroll
                for (int i = 0; i < 4; i++) split_pair(wr[2 * i * kFtCols], wr[(2 * i + 1) * kFtCols], p0[i], p1[i], p2[i], rest);
            }
            const uint32_t t_w = t_lane + kFtPieces + (uint32_t)((s & 1) * 48 + part * 4);
            tmem_st4(t_w, p0);
            tmem_st4(t_w + 16, p1);
            tmem_st4(t_w + 32, p2);
            const unsigned char* xr = raw + kFtRawW + row0 * 128 + quad * 16;
            unsigned char* xs = smem_raw + (s & 1) * 2 * kFtTile;
            // all token groups at a time, so that their latencies overlap; the 8 rows of a warp's group are there or not: nt is a multiple of 16
            float4 v[kFtTok / 64];
#pragma unroll
            for (int j = 0; j < kFtTok / 64; j++)
                v[j] = (warp >> 1) * 8 + 64 * j < nt ? *reinterpret_cast<const float4*>(xr + j * 8192) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int j = 0; j < kFtTok / 64; j++) {
                uint2 q0, q1, q2;
                split_pair(v[j].x, v[j].y, q0.x, q1.x, q2.x, rest);
                split_pair(v[j].z, v[j].w, q0.y, q1.y, q2.y, rest);
                if ((warp >> 1) * 8 + 64 * j < nt) {
                    *reinterpret_cast<uint2*>(xs + x_at + j * 8192) = q0;
                    *reinterpret_cast<uint2*>(xs + (x_at ^ 64u) + j * 8192) = q1;  // 16-byte chunk + 4, swizzled
                    *reinterpret_cast<uint2*>(xs + kFtTile + x_at + j * 8192) = q2;
                }
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(full0 + 8 * (s & 1));
            if (++slot == kFtDepth) {
                slot = 0;
                phase ^= 1;
            }
            if (s > 0) ok = add(s - 1);
        }
        if (ok) ok = add(n_stages - 1);
        lossy = (rest & 0xffffu) != 0u;
    }
    pdl_launch_dependents();

    // A result stands if it is finite and so large that what its operands lost does not count; if one of a block's does not, the
    // block computes all of its results again.
    const int ks = gridDim.y, q = warp & 3;
    float* again = reinterpret_cast<float*>(smem_raw + kFtPiecesBytes);
    auto stands = [](float v, float least, bool whole) { return (fabsf(v) >= least && isfinite(v)) || (whole && v == 0.f); };
    auto least_of = [&](float top) { return fmaxf(kFtLeast, top * ((float)a.K * kFtLost)); };
    const bool fine = __syncthreads_and(ok);  // every warp has seen the last products: the operands are not read any more
    if (ks > 1) cluster_wait();               // the other ranks have s_top
    if (!fine) {
        if (warp == kFtWarps) {
            ring_drain(raw0, kFtDepth, loaded);
            ring_drain(done0, 2, issued);
        }
        if (tid < ks) atomicMax(cluster.map_shared_rank(&s_top, tid), kGaveUp);
    } else if (__syncthreads_or(lossy)) {
        const unsigned top = __float_as_uint(largest<NK>(a, m0, m_rows, n0, k_begin, k_end));
        const unsigned most = __reduce_max_sync(0xffffffffu, top);
        if (lane < ks) atomicMax(cluster.map_shared_rank(&s_top, lane), most);
    }
    if (ks == 1) __syncthreads();
    if (ks == 1) {
        const int n = n0 + q * 32 + lane;
        const float top = __uint_as_float(s_top), least = least_of(top);
        bool bad = false;
        if (fine && warp < kFtWarps && n < a.N) {
#pragma unroll
            for (int i = 0; i < 3 * kFtGroup; i++)
                if (i < np && part * np + i < m_rows) bad |= !stands(acc[i], least, top == 0.f);
        }
        if (__syncthreads_or(bad)) {
            plain_tile<NK>(a, again, m0, m_rows, n0);
        } else if (fine && warp < kFtWarps && n < a.N) {
#pragma unroll
            for (int i = 0; i < 3 * kFtGroup; i++)
                if (i < np && part * np + i < m_rows) finish_f32(a, m0 + part * np + i, n, acc[i]);
        }
    } else {
        float* red = reinterpret_cast<float*>(smem_raw);  // [nt][128]
        if (fine && warp < kFtWarps) {
#pragma unroll
            for (int i = 0; i < 3 * kFtGroup; i++)
                if (i < np) red[(part * np + i) * kFtCols + q * 32 + lane] = acc[i];
        }
        cluster.sync();
        // this rank's tokens; their sums go into its own buffer, in the place that no other rank reads
        const float top = __uint_as_float(s_top);
        const int tokens = s_top == kGaveUp ? 0 : m_rows;  // a rank that gave up: nothing of the tile is stored
        const int rank = blockIdx.y, per = (tokens + ks - 1) / ks, r0 = min(rank * per, tokens), r1 = min(r0 + per, tokens);
        const float least = least_of(top);
        bool bad = false;
        for (int e = r0 * kFtCols + tid; e < r1 * kFtCols; e += kFtThreads) {
            float p[8];
#pragma unroll
            for (int r = 0; r < 8; r++) p[r] = r < ks ? cluster.map_shared_rank(red, r)[e] : 0.f;
            float v = p[0];
#pragma unroll
            for (int r = 1; r < 8; r++) v += p[r];
            red[e] = v;
            bad |= n0 + e % kFtCols < a.N && !stands(v, least, top == 0.f);
        }
        if (__syncthreads_or(bad)) {
            plain_tile<NK>(a, again, m0 + r0, r1 - r0, n0);
        } else {
            for (int e = r0 * kFtCols + tid; e < r1 * kFtCols; e += kFtThreads) {
                const int n = n0 + e % kFtCols;
                if (n < a.N) finish_f32(a, m0 + e / kFtCols, n, red[e]);
            }
        }
        cluster.sync();  // peers may still be reading this block's sums
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}
static const TimeoutFlag timeout_flag(tc_flag_read_clear, tc_flag_address);

template <bool NK>
static cudaLaunchConfig_t ft_config(dim3 grid, cudaStream_t st, cudaLaunchAttribute (&at)[2])
{
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 1;
    at[0].val.clusterDim.y = grid.y;
    at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(kFtThreads);
    cfg.dynamicSmemBytes = kFtSmem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    return cfg;
}

// Blocks of clusters of `ks` that are resident at once, asked once per device.
template <bool NK>
static int ft_slots(int ks)
{
    static std::mutex mu;
    static int known[kMaxDevices][9] = {};
    std::lock_guard<std::mutex> lock(mu);
    int& n = known[current_device()][ks];
    if (n == 0) {
        cudaLaunchAttribute at[2];
        cudaLaunchConfig_t cfg = ft_config<NK>(dim3(1024, ks, 1), nullptr, at);
        cfg.numAttrs = 1;
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, gemm_f32_tc_kernel<NK>, &cfg) != cudaSuccess || clusters < 1) {
            (void)cudaGetLastError();
            clusters = num_sms() / ks;
        }
        n = std::max(1, clusters) * ks;
    }
    return n;
}

template <bool NK>
static cudaError_t launch_ft(const GemmF32& a, cudaStream_t st)
{
    auto kern = gemm_f32_tc_kernel<NK>;
    static DeviceOnce attr;
    const cudaError_t e = attr.run([kern] {
        const cudaError_t r = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kFtSmem);
        return r != cudaSuccess ? r : prefer_max_shared((const void*)kern);
    });
    if (e != cudaSuccess) return e;
    // Tokens per block and K split by an estimate: waves of blocks x (stages of a block x time of a stage + what a block costs
    // besides, both in cycles, fitted to 80 and 176 tokens).
    const int cols = (a.N + kFtCols - 1) / kFtCols, total = (a.K + kFtK - 1) / kFtK, z_least = (a.M + kFtTok - 1) / kFtTok;
    int best_nt = 0, best_per = 0, best_ks = 1;
    double best = 0.0;
    for (int z = z_least; z <= z_least + 2; z++) {
        const int nt = ((a.M + z - 1) / z + 15) / 16 * 16, blocks_z = (a.M + nt - 1) / nt;
        for (int ks = 1; ks <= std::min(8, total); ks++) {
            const int per = (total + ks - 1) / ks;
            if (per * (ks - 1) >= total) continue;
            const long slots = ft_slots<NK>(ks), blocks = (long)cols * blocks_z * ks;
            const double cost = (double)((blocks + slots - 1) / slots) * (per * (1400.0 + 5.7 * nt) + 5000.0 + (ks > 1 ? 4000.0 : 0.0));
            if (best_nt == 0 || cost < best) {
                best = cost;
                best_nt = nt;
                best_per = per;
                best_ks = ks;
            }
        }
    }
    const long z = (a.M + best_nt - 1) / best_nt;
    CUtensorMap map_x, map_w;
    if (make_map_f32(&map_x, a.x, a.K, a.M, a.ldx, kFtK, best_nt, false) != ONELLM_OK ||
        make_map_f32(&map_w, a.W, NK ? a.K : a.N, NK ? a.N : a.K, a.ldw, NK ? kFtK : kFtCols, NK ? kFtCols : kFtK, NK) != ONELLM_OK)
        return cudaErrorInvalidValue;
    cudaLaunchAttribute at[2];
    const cudaLaunchConfig_t cfg = ft_config<NK>(dim3(cols, best_ks, (unsigned)z), st, at);
    note_launch();
    return cudaLaunchKernelEx(&cfg, kern, a, map_x, map_w, best_nt, best_per);
}

// Below, the chain of sgemm_kernel is as close or closer for some operands (equal ones, ones of very unequal size); from here on this
// kernel is the closer for every kind that was tried.  256 products, error against 64 bits of the chain | here: normal 2.9e-7 | 8.0e-8,
// positive 2.2e-7 | 7.0e-8, log-normal 8.7e-8 | 5.7e-8, all equal 1.19e-7 | 1.16e-7.
constexpr int kFtLeastK = 256;

// Sizes, strides and alignment it covers: 16-byte rows.
bool gemm_f32_tc_takes(const GemmF32& a)
{
    return a.M > kF32SkinnyTokens && a.K >= kFtLeastK && a.K % 4 == 0 && a.ldx % 4 == 0 && a.ldw % 4 == 0 && (a.w_nk || a.N % 4 == 0) &&
           aligned16(a.x) && aligned16(a.W) && ((long)a.M + 15) / 16 <= 65535;
}

cudaError_t gemm_f32_tc(const GemmF32& a, cudaStream_t st) { return a.w_nk ? launch_ft<true>(a, st) : launch_ft<false>(a, st); }

}  // namespace onellm
