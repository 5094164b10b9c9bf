// Context-phase projections (M > 64 tokens) on the 5th-generation tensor cores of sm_100a.
//
// Replaces the cuBLAS GEMM behind launchLinearGemm (src/kernels/qkv_linear.cu:8-65,
// src/kernels/cublas_wrapper.cc:45-90 of the reference) for prefill shapes: y[M,N] = x[M,K] . W with
// W [K,N] (the layer weights, N contiguous) or W [N,K] (the LM head), fp16 in, fp32 accumulate.
//
// Persistent: one block per SM walks 128 x 256 output tiles (with 128 x 128 tiles the operand traffic from L2
// into shared memory, 15.6 KB per MFLOP, was what bounded the kernel; the wider tile needs 11.7) in an order
// that keeps the tiles in flight on a near-square patch of the output.  Warp 0 streams 64-deep K slices of
// both operands into a ring of four shared-memory stages with TMA (cp.async.bulk.tensor, 128-byte swizzle; no
// cluster multicast anywhere); one thread of warp 1 issues tcgen05.mma (M = 128, N = 256, K = 16, kind::f16)
// and releases each stage with tcgen05.commit; tensor memory holds two 256-column accumulators, so warps 2-5
// (tcgen05.ld, convert, store) drain tile i while the MMAs of tile i + 1 run.
// Where it is the faster (persistent_us) two blocks work as a pair on a tile of 256 rows (cta_group::2): an SM then takes in 32 KB
// a slice instead of 48, the operand traffic being what bounds the single form (128 x 256: 0.40 us a slice, pairs 0.37, which is
// 1.54 PFLOP/s on long prompts).
// The [K,N] weight is used as it lies in memory: it is the "MN-major" B operand of the MMA
// (four 64-column TMA boxes per stage), so no transposed copy of the weights is ever made.
// Every wait on an mbarrier is bounded; on a time-out the block records it in a device flag,
// skips its stores, frees its tensor memory and exits.
#include <cooperative_groups.h>
#include <cuda.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>

#include "project.h"
#include "tc_common.cuh"

namespace cg = cooperative_groups;

namespace onellm {

constexpr int kTcBM = 128, kTcBN = 256, kTcBK = 64;
constexpr int kTcStages = 4;
constexpr int kTcPairStages = 6;     // of 32 KB: the same shared memory
constexpr int kTcBand = 16;  // row tiles per band of the tile order
constexpr int kTcThreads = 192;      // producer warp, MMA warp, four epilogue warps
constexpr int kTcEpiThreads = 128;
constexpr int kTcATile = kTcBM * kTcBK * 2;        // 16 KB: 128 rows x 128 bytes
constexpr int kTcBTile = kTcBN * kTcBK * 2;        // 32 KB: [K,N] four boxes of 64 k-rows x 128 bytes; [N,K] 256 rows x 128 bytes
constexpr int kTcBChunk = 64 * kTcBK * 2;          // 8 KB: one 64-column chunk of a [K,N] stage
constexpr int kTcStageBytes = kTcATile + kTcBTile;
constexpr int kTcTurnBytes = 32 * 32 * 4;  // a warp's 32 x 32 values on their way to memory
constexpr int kTcSmemBytes = kTcStages * kTcStageBytes + 1024 /* alignment slack */ + 256 /* barriers, TMEM address */ + kTcEpiThreads / 32 * kTcTurnBytes;

// W_NK = false: W [K,N] (B operand MN-major);  W_NK = true: W [N,K] (B operand K-major).
// Persistent: grid = min(tiles, SMs) blocks of six warps; block c works on tiles c, c + grid, ... in band
// order (see below).  Warp 0 (one thread) is the TMA producer, warp 1 (one thread) issues the MMAs,
// warps 2-5 are the epilogue.  Tensor memory holds TWO 128 x 256 accumulators, so the MMAs of the next
// tile run while the epilogue warps drain the previous one.
// MODE 2: two [K,N] weights; the 256 accumulator columns of a tile are 128 columns of x.W (gate) beside the
// same 128 columns of x.W2 (up), and the epilogue stores silu(gate) * up: the gate GEMM, the up GEMM and
// launchAct of src/layers/ffn/ffn.cpp:62-66 in one pass, without the [T, 2, I] buffer.
// Epilogue options that let the context phase run without norm kernels, as the decode step does (the norm's gamma
// is multiplied into the weight rows beforehand):
//   row_ss:  sums of squares of the rows of x, as ss_parts partial sums per row; the result rows are scaled by
//            rsqrt(sum / K + eps), i.e. this is the projection of RMSNorm(x)
//   resid:   y = resid + bias + result (resid may be y itself: an element is read and written by the same thread)
//   ss_out:  [M, ceil(N / tile columns)]: the sum of squares of the stored (rounded) values of each row inside this
//            tile's columns -- the row_ss of the projection that reads y next.  Every entry is written by exactly
//            one block, so the sums do not depend on the order the blocks run in.
//   act:     gate function of MODE 2
//   ldy:     row stride of y (and of resid); 0: N
//   f32:     y and resid are float instead of the element type (no ss_out then)
//   scale:   with f32, factor on the result in front of the residual
//   limit:   bound of the clamped gate function
// GROUPED: the rows of x and y lie in groups with weights of their own (onellm_row_groups: the experts of a mixture).  The
// row tiles come from a table, 128 rows of one group each; the weights are stacked, so that a tile reads K rows of W from
// row group * K on.  Columns of x behind K are zero-filled, so that a last K slice that reaches into the next weight adds
// nothing.
struct TcEpilogue {
    const float* row_ss;
    int ss_parts;
    float eps;
    const void* resid;
    const void* bias;
    float* ss_out;
    int act;
    long ldy;
    int f32;
    float scale = 1.f, limit = 0.f;
};

// PAIR: the two blocks of a cluster share a tile of 256 rows (cta_group::2): a block loads its 128 rows of x and half the columns of W
// (two weights: one of them), 32 KB a slice instead of 48, and finishes its rows.
template <typename T, int MODE, bool GROUPED = false, bool PAIR = false>
__global__ void __launch_bounds__(kTcThreads)
gemm_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
               const __grid_constant__ CUtensorMap map_b2, T* y, int M, int N, int K, const TcEpilogue epi, const RowGroups grp)
{
    constexpr bool W_NK = MODE == 1;
    constexpr bool DUAL = MODE == 2;
    constexpr int kOutN = DUAL ? kTcBN / 2 : kTcBN;  // output columns per tile
    static_assert(!(PAIR && GROUPED), "the tiles of groups have 128 rows");
    constexpr int kStages = PAIR ? kTcPairStages : kTcStages, kStageBytes = kTcATile + (PAIR ? kTcBTile / 2 : kTcBTile);
    constexpr int kTileM = PAIR ? 2 * kTcBM : kTcBM, kBand = PAIR ? kTcBand / 2 : kTcBand;
    const uint32_t rank = PAIR ? (uint32_t)cg::this_cluster().block_rank() : 0u;
    const int tile0 = PAIR ? (int)blockIdx.x >> 1 : (int)blockIdx.x, tile_step = PAIR ? (int)gridDim.x >> 1 : (int)gridDim.x;
    extern __shared__ unsigned char smem_raw[];
    // 1024-byte alignment for the 128-byte swizzle pattern
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kStages * kStageBytes);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kStages + 4);
    const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + kStages);
    const uint32_t acc_full0 = smem_u32(bars + 2 * kStages), acc_empty0 = smem_u32(bars + 2 * kStages + 2);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // Tile order: the linear tile index walks down a band of kTcBand row tiles, then moves one column
    // tile to the right, so the tiles in flight at one time (one per SM) cover a near-square patch
    // of the output and share their A row blocks and B column blocks in L2.  (Row-major order made every
    // wave touch all column tiles of B: operands were read from DRAM seven times over.)
    int tiles_m = (M + kTileM - 1) / kTileM;
    const int tiles_n = (N + kOutN - 1) / kOutN;
    int n_tiles = tiles_m * tiles_n;
    // first row and column of a tile, the row of the stacked weights it starts at, the end of its rows
    auto tile_origin = [&](int t, int& m0, int& n0, int& k0, int& m_end) {
        const int per_band = kBand * tiles_n;
        const int band = t / per_band, in_band = t % per_band;
        const int band_rows = min(kBand, tiles_m - band * kBand);
        const int mt = band * kBand + in_band % band_rows;
        n0 = (in_band / band_rows) * kOutN;
        if constexpr (GROUPED) {
            const int g = grp.tile_group[mt];
            m0 = grp.tile_row[mt];
            k0 = g * K;
            m_end = grp.off[g + 1];
        } else {
            m0 = mt * kTileM + (int)rank * kTcBM;
            k0 = 0;
            m_end = M;
        }
    };
    const int k_steps = (K + kTcBK - 1) / kTcBK;
    const uint32_t ring = smem_u32(smem);

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; s++) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(empty0 + 8 * s, 1);
        }
        for (int a = 0; a < 2; a++) {
            mbar_init(acc_full0 + 8 * a, 1);
            mbar_init(acc_empty0 + 8 * a, PAIR ? 2 * kTcEpiThreads / 32 : kTcEpiThreads);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) {
        if constexpr (PAIR) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(2u * kTcBN) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(2u * kTcBN) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if constexpr (PAIR) cg::this_cluster().sync();  // the other block's barriers
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;

    pdl_wait();  // x comes from the previous kernel in the stream
    if constexpr (GROUPED) {
        tiles_m = *grp.n_tiles;
        n_tiles = tiles_m * tiles_n;
    }

    bool ok = true;
    int used = 0;  // warp 0: stages it has loaded, warp 1: stages its products read
    if (warp == 0) {
        // producer: one 64-deep slice of A and of B per stage, tile after tile
        const bool leader = elect_one();
        uint32_t s = 0, round = 0;
        for (int t = tile0; t < n_tiles && ok; t += tile_step) {
            int m0, n0, k0, m_end;
            tile_origin(t, m0, n0, k0, m_end);
            for (int ks = 0; ks < k_steps; ks++) {
                if (round > 0) ok = mbar_wait_warp(empty0 + 8 * s, (round - 1) & 1);
                if (!ok) break;
                if (PAIR && leader) {
                    const uint32_t bar = map_to_rank(full0 + 8 * s, 0), a_dst = ring + s * kStageBytes, b_dst = a_dst + kTcATile;
                    if (rank == 0) mbar_expect_tx(full0 + 8 * s, 2 * kStageBytes);  // what both blocks load
                    tma_load_2d_pair(a_dst, &map_a, ks * kTcBK, m0, bar);
                    if (W_NK) {
                        tma_load_2d_pair(b_dst, &map_b, ks * kTcBK, n0 + (int)rank * (kTcBN / 2), bar);
                    } else {
                        // one weight: the 128 columns of this rank; two: the rank's weight
                        const int n = DUAL ? n0 : n0 + (int)rank * (kTcBN / 2);
#pragma unroll
                        for (int c = 0; c < 2; c++)
                            tma_load_2d_pair(b_dst + c * kTcBChunk, DUAL && rank == 1 ? &map_b2 : &map_b, n + 64 * c, ks * kTcBK, bar);
                    }
                } else if (leader) {
                    const uint32_t bar = full0 + 8 * s, a_dst = ring + s * kStageBytes, b_dst = a_dst + kTcATile;
                    mbar_expect_tx(bar, kStageBytes);
                    tma_load_2d(a_dst, &map_a, ks * kTcBK, m0, bar);
                    if (W_NK) {
                        tma_load_2d(b_dst, &map_b, ks * kTcBK, n0, bar);
                    } else if (DUAL) {
#pragma unroll
                        for (int c = 0; c < 2; c++) {
                            tma_load_2d(b_dst + c * kTcBChunk, &map_b, n0 + 64 * c, k0 + ks * kTcBK, bar);
                            tma_load_2d(b_dst + (2 + c) * kTcBChunk, &map_b2, n0 + 64 * c, k0 + ks * kTcBK, bar);
                        }
                    } else {
#pragma unroll
                        for (int c = 0; c < kTcBN / 64; c++) tma_load_2d(b_dst + c * kTcBChunk, &map_b, n0 + 64 * c, k0 + ks * kTcBK, bar);
                    }
                }
                if (++s == kStages) {
                    s = 0;
                    round++;
                }
            }
        }
        used = (int)(round * kStages + s);
        if (PAIR && rank == 1) pdl_launch_dependents();
    } else if (warp == 1 && rank == 0) {
        // instruction descriptor: D = f32, A and B of type T, A K-major, B MN-major unless W_NK, N = 256, M = 128 (256 of a pair)
        const uint32_t idesc = (1u << 4) | umma_operand_bits<T>() | ((W_NK ? 0u : 1u) << 16) | ((uint32_t)(kTcBN >> 3) << 17) | ((uint32_t)(kTileM >> 4) << 24);
        // A: K-major, rows of 128 bytes, 8-row groups 1024 bytes apart; 16 k = 32 bytes further in the row
        // B [N,K]: same form.  B [K,N]: MN-major, 64-column chunks 8192 bytes apart (LBO), 8-row k groups
        // 1024 bytes apart (SBO); 16 k = two groups further
        // These are the descriptors of the first stage; a stage or a step inside it adds (bytes >> 4) to the address field.
        const uint64_t da = umma_desc(ring, 16, 1024), db = umma_desc(ring + kTcATile, W_NK ? 16 : kTcBChunk, 1024);
        const bool leader = elect_one();
        int lt = 0;
        uint32_t s = 0, phase = 0;
        for (int t = tile0; t < n_tiles && ok; t += tile_step, lt++) {
            const int acc = lt & 1, use = lt >> 1;
            // the accumulator must have been drained by the epilogue of the tile that used it before
            if (use >= 1) ok = mbar_wait_warp(acc_empty0 + 8 * acc, (use - 1) & 1);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t tmem_d = tmem_base + (uint32_t)(acc * kTcBN);
            for (int ks = 0; ks < k_steps; ks++) {
                ok = mbar_wait_warp(full0 + 8 * s, phase);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (leader) {
                    const uint64_t at = (uint64_t)(s * (kStageBytes >> 4));
#pragma unroll
                    for (int kk = 0; kk < kTcBK / 16; kk++) {
                        const uint64_t ad = da + at + (uint64_t)((kk * 32) >> 4), bd = db + at + (uint64_t)((W_NK ? kk * 32 : kk * 2048) >> 4);
                        if constexpr (PAIR) umma_f16_pair(tmem_d, ad, bd, idesc, (ks > 0 || kk > 0) ? 1u : 0u);
                        else umma_f16(tmem_d, ad, bd, idesc, (ks > 0 || kk > 0) ? 1u : 0u);
                    }
                    // frees the stage when these MMAs have read it
                    if constexpr (PAIR) umma_commit_pair(empty0 + 8 * s);
                    else umma_commit(empty0 + 8 * s);
                }
                __syncwarp();
                used++;
                if (++s == kStages) {
                    s = 0;
                    phase ^= 1;
                }
            }
            if (ok && leader) {  // the tile is complete when everything issued so far has run
                if constexpr (PAIR) umma_commit_pair(acc_full0 + 8 * acc);
                else umma_commit(acc_full0 + 8 * acc);
            }
        }
        pdl_launch_dependents();
    } else if (warp >= 2) {
        // epilogue: warp w may touch TMEM lanes 32 * (w % 4) .. + 31, which are the tile rows of the same numbers
        const int q = warp & 3;
        const size_t ldy = epi.ldy ? (size_t)epi.ldy : (size_t)N;
        float4* turn = reinterpret_cast<float4*>(smem + kStages * kStageBytes + 256 + (warp - 2) * kTcTurnBytes);
        auto turned = [&](int r, int chunk) { return turn + r * 8 + (chunk ^ (r & 7)); };  // 16 bytes of row r, free of bank conflicts both ways
        int lt = 0;
        for (int t = tile0; t < n_tiles && ok; t += tile_step, lt++) {
            const int acc = lt & 1, use = lt >> 1;
            int m0, n0, k0, m_end;
            tile_origin(t, m0, n0, k0, m_end);
            // In memory a lane has 16 bytes of a row: of every fourth row (f32), of every eighth (16-bit elements)
            const int r_step = epi.f32 ? 4 : 8, r_lane = epi.f32 ? lane >> 3 : lane >> 2, c_lane = epi.f32 ? (lane & 7) * 4 : (lane & 3) * 8;
            const int m_lane = m0 + q * 32 + r_lane, n_lane = n0 + c_lane, turns = 32 / r_step, size = epi.f32 ? 4 : (int)sizeof(T);
            auto inside = [&](int c0, int i) { return m_lane + i * r_step < m_end && n_lane + c0 < N; };  // N is a multiple of 8
            auto element = [&](int c0, int i) { return ((size_t)(m_lane + i * r_step) * ldy + n_lane + c0) * size; };
            uint4 rs[8];  // the residual of the next 32 columns, asked for one turn ahead
            auto fetch = [&](int c0) {
#pragma unroll
                for (int i = 0; i < 8; i++)
                    if (i < turns && c0 < kOutN && inside(c0, i)) rs[i] = *reinterpret_cast<const uint4*>(static_cast<const unsigned char*>(epi.resid) + element(c0, i));
            };
            if (epi.resid) fetch(0);
            ok = mbar_wait(acc_full0 + 8 * acc, use & 1);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int row = m0 + q * 32 + lane;
            const bool row_ok = row < m_end;
            float inv = 1.f, sq[4] = {0.f, 0.f, 0.f, 0.f};
            const bool scaled = GROUPED ? grp.row_scale != nullptr : epi.row_ss != nullptr;
            if (GROUPED && scaled && row_ok) inv = grp.row_scale[row];
            if (epi.row_ss && row_ok) {
                float ssum = 0.f;
                for (int pp = 0; pp < epi.ss_parts; pp++) ssum += epi.row_ss[(size_t)row * epi.ss_parts + pp];
                inv = rsqrtf(ssum / (float)K + epi.eps);
            }
#pragma unroll 1
            for (int c0 = 0; c0 < kOutN; c0 += 32) {
                uint32_t r[32];
                tmem_ld32(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * kTcBN + c0), r);
                if (DUAL) {
                    uint32_t u[32];
                    tmem_ld32(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * kTcBN + kOutN + c0), u);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    gate_row(reinterpret_cast<float(&)[32]>(r), reinterpret_cast<const float(&)[32]>(u), inv, epi.act, epi.limit);
                } else {
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (scaled) {
#pragma unroll
                        for (int i = 0; i < 32; i++) r[i] = __float_as_uint(__uint_as_float(r[i]) * inv);
                    }
                }
                // A lane has a row of the accumulator; written from there, every store of a warp would touch 32 lines (2000 tokens, K 9728, 2048
                // float outputs on top of a residual: 20 us behind the last product).  Turned around in shared memory, a warp's
                // accesses cover whole 64- or 128-byte parts of rows.
#pragma unroll
                for (int i = 0; i < 8; i++) *turned(lane, i) = make_float4(__uint_as_float(r[4 * i]), __uint_as_float(r[4 * i + 1]), __uint_as_float(r[4 * i + 2]), __uint_as_float(r[4 * i + 3]));
                __syncwarp();
                if (epi.f32) {
                    float a[4] = {0.f, 0.f, 0.f, 0.f};
                    if (epi.bias && n_lane + c0 < N) {
#pragma unroll
                        for (int e = 0; e < 4; e++) a[e] = to_float(static_cast<const T*>(epi.bias)[n_lane + c0 + e]);
                    }
                    const float sc = epi.scale;
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        float4 v = *turned(r_lane + 4 * i, c_lane / 4);
                        if (epi.bias) v.x += a[0], v.y += a[1], v.z += a[2], v.w += a[3];
                        if (epi.resid) {
                            v.x = fmaf(v.x, sc, __uint_as_float(rs[i].x)), v.y = fmaf(v.y, sc, __uint_as_float(rs[i].y));
                            v.z = fmaf(v.z, sc, __uint_as_float(rs[i].z)), v.w = fmaf(v.w, sc, __uint_as_float(rs[i].w));
                        }
                        if (inside(c0, i)) *reinterpret_cast<float4*>(reinterpret_cast<unsigned char*>(y) + element(c0, i)) = v;
                    }
                    if (epi.resid) fetch(c0 + 32);
                } else {
                    float a[8];
                    if (epi.bias && n_lane + c0 < N) Vec16<T>::load(static_cast<const T*>(epi.bias) + n_lane + c0, a);
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        float v[8];
                        *reinterpret_cast<float4*>(v) = *turned(r_lane + 8 * i, c_lane / 4);
                        *reinterpret_cast<float4*>(v + 4) = *turned(r_lane + 8 * i, c_lane / 4 + 1);
                        if (epi.bias) {
#pragma unroll
                            for (int e = 0; e < 8; e++) v[e] += a[e];
                        }
                        if (epi.resid) {
                            float x[8];
                            Vec16<T>::unpack(rs[i], x);
#pragma unroll
                            for (int e = 0; e < 8; e++) v[e] += x[e];
                        }
                        const uint4 packed = Vec16<T>::pack(v);
                        if (inside(c0, i)) {
                            *reinterpret_cast<uint4*>(reinterpret_cast<unsigned char*>(y) + element(c0, i)) = packed;
                            if (epi.ss_out) {
                                Vec16<T>::unpack(packed, v);  // what the next projection will read
#pragma unroll
                                for (int e = 0; e < 8; e++) sq[i] = fmaf(v[e], v[e], sq[i]);
                            }
                        }
                    }
                    if (epi.resid) fetch(c0 + 32);
                }
                __syncwarp();
            }
            if (epi.ss_out) {
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    sq[i] += __shfl_xor_sync(0xffffffffu, sq[i], 1);
                    sq[i] += __shfl_xor_sync(0xffffffffu, sq[i], 2);
                    if ((lane & 3) == 0 && m_lane + 8 * i < m_end) epi.ss_out[(size_t)(m_lane + 8 * i) * tiles_n + n0 / kOutN] = sq[i];
                }
            }
            // this thread's reads of the accumulator are over: hand it back to the MMA warp
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            if constexpr (PAIR) {
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(map_to_rank(acc_empty0 + 8 * acc, 0));
            } else {
                mbar_arrive(acc_empty0 + 8 * acc);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if (!__syncthreads_and(ok)) {
        // loads of a pair report to its even block, and the products are its own
        if (warp <= 1 && rank == 0) ring_drain(warp == 0 ? full0 : empty0, kStages, used);
        __syncthreads();
    }
    if constexpr (PAIR) cg::this_cluster().sync();  // neither leaves while the other may reach its barriers or tensor memory
    if (warp == 2) {
        if constexpr (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(2u * kTcBN) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(2u * kTcBN) : "memory");
    }
}

// ---- few tiles: K split over a cluster -------------------------------------------------------------
// The persistent kernel gives a 128 x 256 tile to one SM, so a prompt of a few hundred tokens leaves most of them idle (238
// tokens, 4096 outputs: 32 tiles on 148 SMs).  Here tiles have 128 x 128 outputs (two weights: 64 of each), the blocks of a cluster
// take a K range of one tile each and add their accumulators through distributed shared memory, in rank order; an output row
// of the tile is finished by one warp.  A block has half an SM's shared memory, so that two of them hide each other's start,
// sum and end.
// What bounds it (stamps of %globaltimer, 238 tokens): 1.4 us from a block's start to its first product, 0.8 us to move the
// accumulator, 0.7 us for the cluster to meet; distributed shared memory brings about 14 bytes per cycle and SM, so that a sum
// over four ranks of a 128 x 256 tile took 6 to 7 us (tiles of 256 columns: 19.3 us for o_proj against 15.6), and an SM takes in
// about 60 bytes per cycle of operands.
// Same operands, descriptors, epilogue options and row statistics as gemm_tc_kernel; the K ranges are added in float.
// Measured beside the persistent kernel, 7B shape, 70 | 238 tokens: o_proj 28.9 -> 12.5 | 29.3 -> 15.6 us, down 65.2 -> 23.8 |
// 66.2 -> 28.9, QKV 31.8 -> 24.5 | 33.1 (stays; 29.8 in pairs), 32 outputs (a router) 21.8 -> 6.1 | 21.5 -> 7.2.
constexpr int kSplitBN = 128;
constexpr int kSplitStage = kTcATile + kSplitBN * kTcBK * 2;
constexpr int kSplitStages = 3;
constexpr int kSplitSmem = kSplitStages * kSplitStage + 1024 /* alignment slack */ + 256 /* barriers, TMEM address */;
constexpr int kSplitLd = kSplitBN + 4;  // row stride (floats) of the accumulator in shared memory: rows 16 bytes apart modulo the banks
static_assert(kTcBM * kSplitLd * 4 <= kSplitStages * kSplitStage, "the accumulator takes the place of the ring");
constexpr int kSplitThreads = 320;  // producer warp, MMA warp, eight warps that move the accumulator; all of them add up rows

// grid (column tiles * row tiles, KS), cluster (1 or 2, KS): two column tiles per cluster when ss_out is asked for, which is
// kept per 256 columns
template <typename T, int MODE>
__global__ void __launch_bounds__(kSplitThreads, 2)
gemm_tc_split_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                     const __grid_constant__ CUtensorMap map_b2, T* y, int M, int N, int K, const TcEpilogue epi, int tiles_n, int slices_per_block)
{
    constexpr int BN = kSplitBN;
    constexpr bool W_NK = MODE == 1;
    constexpr bool DUAL = MODE == 2;
    constexpr int kOutN = DUAL ? BN / 2 : BN;
    constexpr int NV = BN / 32;                    // accumulator values of a lane in the epilogue
    constexpr int kLaneCols = kOutN / 32;          // output columns of a lane
    using Floats = typename std::conditional<DUAL, float2, float4>::type;  // a lane's part of a row, in float
    using Halves = typename std::conditional<DUAL, uint32_t, uint2>::type;  // and in T
    static_assert(sizeof(Floats) == kLaneCols * sizeof(float), "the stores of a lane");
    extern __shared__ unsigned char smem_raw[];
    __shared__ float s_sq[kTcBM];
    __shared__ int s_gave_up;
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kSplitStages * kSplitStage);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kSplitStages + 1);
    const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + kSplitStages), acc_full = smem_u32(bars + 2 * kSplitStages);
    cg::cluster_group cluster = cg::this_cluster();
    const int ks = gridDim.y, rank = blockIdx.y;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_tile = blockIdx.x % tiles_n, m0 = (blockIdx.x / tiles_n) * kTcBM, n0 = n_tile * kOutN;
    const uint32_t ring = smem_u32(smem);
    const int slices = (K + kTcBK - 1) / kTcBK;
    const int first = min(rank * slices_per_block, slices), n_slices = min(slices_per_block, slices - first);

    if (threadIdx.x == 0) {
        for (int s = 0; s < kSplitStages; s++) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(empty0 + 8 * s, 1);
        }
        mbar_init(acc_full, 1);
        s_gave_up = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"((uint32_t)BN) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    cluster_arrive();

    pdl_wait();
    bool ok = true;
    int loaded = 0;
    if (warp == 0) {
        const bool leader = elect_one();
        uint32_t s = 0, round = 0;
        for (int it = 0; it < n_slices && ok; it++) {
            if (round > 0) ok = mbar_wait_warp(empty0 + 8 * s, (round - 1) & 1);
            if (ok && leader) {
                const int k = (first + it) * kTcBK;
                const uint32_t bar = full0 + 8 * s, a_dst = ring + s * kSplitStage, b_dst = a_dst + kTcATile;
                mbar_expect_tx(bar, kSplitStage);
                if (W_NK) {
                    tma_load_2d(b_dst, &map_b, k, n0, bar);
                } else if (DUAL) {
#pragma unroll
                    for (int c = 0; c < kOutN / 64; c++) {
                        tma_load_2d(b_dst + c * kTcBChunk, &map_b, n0 + 64 * c, k, bar);
                        tma_load_2d(b_dst + (kOutN / 64 + c) * kTcBChunk, &map_b2, n0 + 64 * c, k, bar);
                    }
                } else {
#pragma unroll
                    for (int c = 0; c < BN / 64; c++) tma_load_2d(b_dst + c * kTcBChunk, &map_b, n0 + 64 * c, k, bar);
                }
                tma_load_2d(a_dst, &map_a, k, m0, bar);
            }
            loaded += ok;
            if (++s == kSplitStages) {
                s = 0;
                round++;
            }
        }
    } else if (warp == 1) {
        const uint32_t idesc = (1u << 4) | umma_operand_bits<T>() | ((W_NK ? 0u : 1u) << 16) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(kTcBM >> 4) << 24);
        // descriptors of the first stage; a stage or a step inside it adds (bytes >> 4) to the address field
        const uint64_t da = umma_desc(ring, 16, 1024), db = umma_desc(ring + kTcATile, W_NK ? 16 : kTcBChunk, 1024);
        const bool leader = elect_one();
        uint32_t s = 0, phase = 0;
        for (int it = 0; it < n_slices && ok; it++) {
            ok = mbar_wait_warp(full0 + 8 * s, phase);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (ok && leader) {
                const uint64_t at = (uint64_t)(s * (kSplitStage >> 4));
#pragma unroll
                for (int kk = 0; kk < kTcBK / 16; kk++)
                    umma_f16(tmem_base, da + at + (uint64_t)((kk * 32) >> 4), db + at + (uint64_t)((W_NK ? kk * 32 : kk * 2048) >> 4), idesc,
                             (it > 0 || kk > 0) ? 1u : 0u);
                umma_commit(empty0 + 8 * s);
            }
            __syncwarp();
            if (++s == kSplitStages) {
                s = 0;
                phase ^= 1;
            }
        }
        if (leader) umma_commit(acc_full);  // arrives when everything issued has run (also when the loop gave up)
        pdl_launch_dependents();
    }
    __syncwarp();  // the barriers below are warp-wide
    if (warp >= 2) ok = mbar_wait_warp(acc_full, 0);  // the products have read the ring
    const bool fine = __syncthreads_and(ok);
    cluster_wait();  // the other ranks have s_gave_up
    if (!fine) {     // nothing of the cluster's tiles is stored
        if (warp == 0) ring_drain(full0, kSplitStages, loaded);
        if (threadIdx.x < cluster.num_blocks()) *cluster.map_shared_rank(&s_gave_up, threadIdx.x) = 1;
    }

    float* red = reinterpret_cast<float*>(smem);  // [128][kLd], in place of the ring
    const int rows_per_rank = (kTcBM + ks - 1) / ks;
    const size_t ldy = epi.ldy ? (size_t)epi.ldy : (size_t)N;
    // one output row, this lane's columns of it: what the K ranges add up to -> y
    auto finish_row = [&](int tr, float (&v)[NV]) {
        const int m = m0 + tr;
        if (epi.row_ss) {
            float ssum = 0.f;
            for (int pp = lane; pp < epi.ss_parts; pp += 32) ssum += epi.row_ss[(size_t)m * epi.ss_parts + pp];
            const float inv = rsqrtf(warp_sum(ssum) / (float)K + epi.eps);
#pragma unroll
            for (int e = 0; e < NV; e++) v[e] *= inv;
        }
        const int n = n0 + kLaneCols * lane;
        const bool in = n < N;  // N is a multiple of 8
        const size_t at = (size_t)m * ldy + n;
        float sq = 0.f;
        if (in) {
            if constexpr (DUAL) {
#pragma unroll
                for (int e = 0; e < kLaneCols; e++) v[e] = gate_pair(v[e], v[kLaneCols + e], epi.act, epi.limit);
            }
            if (epi.bias) {
#pragma unroll
                for (int e = 0; e < kLaneCols; e += 2) {
                    const float2 a = unpack2<T>(*reinterpret_cast<const uint32_t*>(static_cast<const T*>(epi.bias) + n + e));
                    v[e] += a.x;
                    v[e + 1] += a.y;
                }
            }
            if (epi.f32) {
                if (epi.resid) {
                    __align__(16) float r[kLaneCols];
                    *reinterpret_cast<Floats*>(r) = *reinterpret_cast<const Floats*>(static_cast<const float*>(epi.resid) + at);
#pragma unroll
                    for (int e = 0; e < kLaneCols; e++) v[e] = fmaf(v[e], epi.scale, r[e]);
                }
                *reinterpret_cast<Floats*>(reinterpret_cast<float*>(y) + at) = *reinterpret_cast<const Floats*>(v);
            } else {
                __align__(8) uint32_t w[kLaneCols / 2];
                if (epi.resid) {
                    *reinterpret_cast<Halves*>(w) = *reinterpret_cast<const Halves*>(static_cast<const T*>(epi.resid) + at);
#pragma unroll
                    for (int e = 0; e < kLaneCols / 2; e++) {
                        const float2 a = unpack2<T>(w[e]);
                        v[2 * e] += a.x;
                        v[2 * e + 1] += a.y;
                    }
                }
#pragma unroll
                for (int e = 0; e < kLaneCols / 2; e++) {
                    w[e] = pack2<T>(v[2 * e], v[2 * e + 1]);
                    const float2 a = unpack2<T>(w[e]);  // what the next projection will read
                    sq = fmaf(a.x, a.x, fmaf(a.y, a.y, sq));
                }
                *reinterpret_cast<Halves*>(y + at) = *reinterpret_cast<const Halves*>(w);
            }
        }
        if (epi.ss_out) {
            sq = warp_sum(sq);
            if (lane == 0) s_sq[tr] = sq;
        }
    };
    if (warp >= 2 && fine) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const int q = warp & 3;  // this warp may touch TMEM lanes 32 q .. 32 q + 31, the rows of the same numbers
        const int half = (warp - 2) >> 2;
        float4* row = reinterpret_cast<float4*>(red + (size_t)(q * 32 + lane) * kSplitLd);
#pragma unroll
        for (int c = 0; c < BN / 2; c += 32) {
            const int c0 = half * (BN / 2) + c;
            uint32_t v[32];
            if (n_slices > 0) {
                tmem_ld32(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)c0, v);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            } else {
#pragma unroll
                for (int i = 0; i < 32; i++) v[i] = 0u;
            }
#pragma unroll
            for (int i = 0; i < 8; i++)
                row[c0 / 4 + i] = make_float4(__uint_as_float(v[4 * i]), __uint_as_float(v[4 * i + 1]), __uint_as_float(v[4 * i + 2]),
                                              __uint_as_float(v[4 * i + 3]));
        }
    }
    cluster.sync();
    const bool gave_up = s_gave_up != 0;
    // This rank's rows, one warp a row, or two where at most four ranks leave room for their loads: all loads are on their
    // way before the first is used.
    const int at_once = ks <= 4 ? 2 : 1;
    const int peer0 = (int)cluster.block_rank() - rank * (int)(cluster.dim_blocks().x);  // rank 0 of this column tile
    const int peer_step = (int)cluster.dim_blocks().x;
    for (int i = warp * at_once; i < rows_per_rank; i += kSplitThreads / 32 * at_once) {
        const int tr = rank * rows_per_rank + i;
        if (tr >= kTcBM || m0 + tr >= M || gave_up) break;
        const bool second = at_once == 2 && i + 1 < rows_per_rank && tr + 1 < kTcBM && m0 + tr + 1 < M;
        float p[8][NV];
        const float* mine = red + (size_t)tr * kSplitLd + kLaneCols * lane;
#pragma unroll
        for (int g = 0; g < 8; g++) {
            const int from = at_once == 2 ? g & 3 : g;
#pragma unroll
            for (int e = 0; e < NV; e++) p[g][e] = 0.f;
            if (from < ks && (at_once == 1 || g < 4 || second)) {
                const float* peer = cluster.map_shared_rank(mine + (at_once == 2 && g >= 4 ? kSplitLd : 0), peer0 + from * peer_step);
                if constexpr (DUAL) {
                    const float2 f = *reinterpret_cast<const float2*>(peer), h = *reinterpret_cast<const float2*>(peer + kOutN);
                    p[g][0] = f.x;
                    p[g][1] = f.y;
                    p[g][2] = h.x;
                    p[g][3] = h.y;
                } else {
                    const float4 f = *reinterpret_cast<const float4*>(peer);
                    p[g][0] = f.x;
                    p[g][1] = f.y;
                    p[g][2] = f.z;
                    p[g][3] = f.w;
                }
            }
        }
        __align__(16) float v[NV], u[NV];
#pragma unroll
        for (int e = 0; e < NV; e++) v[e] = u[e] = 0.f;
#pragma unroll
        for (int g = 0; g < 8; g++)  // rank order
#pragma unroll
            for (int e = 0; e < NV; e++) {
                if (at_once == 2 && g >= 4) u[e] += p[g][e];
                else v[e] += p[g][e];
            }
        finish_row(tr, v);
        if (second) finish_row(tr + 1, u);
    }
    cluster.sync();  // peers may still be reading this block's sums
    if (epi.ss_out) {
        // the row statistics of 256 columns: two tiles side by side in the cluster
        if (n_tile % 2 == 0 && n0 < N && !gave_up)
            for (int i = threadIdx.x; i < rows_per_rank; i += kSplitThreads) {
                const int tr = rank * rows_per_rank + i;
                if (tr >= kTcBM || m0 + tr >= M) break;
                epi.ss_out[(size_t)(m0 + tr) * ((N + kTcBN - 1) / kTcBN) + n_tile / 2] =
                    s_sq[tr] + *cluster.map_shared_rank(&s_sq[tr], (int)cluster.block_rank() + 1);
            }
        __syncwarp();
        cluster.sync();
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 2) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)BN) : "memory");
}

// ---- host side -----------------------------------------------------------------------------------
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                   const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled()
{
    static EncodeTiledFn fn = nullptr;
    static std::mutex mu;
    std::lock_guard<std::mutex> lock(mu);
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}

// 2-D tensor map of 16-bit elements: `inner` contiguous elements, `outer` rows of `inner` elements; box {64, box_outer}; 128-byte swizzle
int make_map(CUtensorMap* map, const void* base, uint64_t inner, uint64_t outer, uint32_t box_outer)
{
    EncodeTiledFn enc = encode_tiled();
    ONELLM_REQUIRE(enc, ONELLM_ERR_CUDA, "gemm: cuTensorMapEncodeTiled is not available from the driver");
    const cuuint64_t dims[2] = {inner, outer};
    const cuuint64_t strides[1] = {inner * sizeof(__half)};
    const cuuint32_t box[2] = {64, box_outer};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    ONELLM_REQUIRE(r == CUDA_SUCCESS, ONELLM_ERR_CUDA, "gemm: cuTensorMapEncodeTiled failed with %d", (int)r);
    return ONELLM_OK;
}

int make_chunk_map(CUtensorMap* map, const void* base, uint64_t inner, uint64_t outer, uint32_t box_rows, uint32_t box_chunks)
{
    EncodeTiledFn enc = encode_tiled();
    ONELLM_REQUIRE(enc, ONELLM_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    const cuuint64_t dims[3] = {64, outer, inner / 64};
    const cuuint64_t strides[2] = {inner * 2, 128};
    const cuuint32_t box[3] = {64, box_rows, box_chunks};
    const cuuint32_t estr[3] = {1, 1, 1};
    const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    ONELLM_REQUIRE(r == CUDA_SUCCESS, ONELLM_ERR_CUDA, "cuTensorMapEncodeTiled failed with %d", (int)r);
    return ONELLM_OK;
}

int make_map_f32(CUtensorMap* map, const void* base, uint64_t inner, uint64_t outer, uint64_t ld, uint32_t box_inner, uint32_t box_outer, bool swizzled)
{
    EncodeTiledFn enc = encode_tiled();
    ONELLM_REQUIRE(enc, ONELLM_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    const cuuint64_t dims[2] = {inner, outer};
    const cuuint64_t strides[1] = {ld * sizeof(float)};
    const cuuint32_t box[2] = {box_inner, box_outer};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           swizzled ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    ONELLM_REQUIRE(r == CUDA_SUCCESS, ONELLM_ERR_CUDA, "cuTensorMapEncodeTiled failed with %d", (int)r);
    return ONELLM_OK;
}

int gemm_f16_skinny(const __half* x, const __half* W, __half* y, int M, int N, int K, int w_layout, cudaStream_t st);

// K split of a projection with few tiles; ks 0: the persistent kernel.
struct SplitPlan {
    int ks, per;
};

// Estimated time in us of the persistent kernel, blocks alone or in pairs, from a sweep over 200 to 3817 tokens and 13 weights: 8 us around
// the slices of 64 k; where no block has a second tile a slice takes 0.335 us, 0.38 when all SMs ask for operands (pairs 0.285 and 0.34),
// else 0.40 (0.37); the weights come in at 6.2 TB/s.  Pairs have half as many tiles of twice the rows, so that a token
// count just above a multiple of 256 or a last wave of few tiles can cost them more than they gain.
// Measured alone | in pairs: 3817 tokens, QKV of the 7B shape 282 | 249 us, gate/up 484 | 445, down 312 | 268; 238 tokens, QKV 33.4 |
// 29.8, gate/up 65 | 56; 2000 tokens, 9728 x 2048 65.2 | 58.6; 1030 tokens, o_proj 31 | 47 (144 tiles, 80 pairs).
static double persistent_us(int M, int N, int K, bool dual, bool pairs)
{
    const long columns = dual ? 2L * N : N, slices = (K + kTcBK - 1) / kTcBK;
    const long rows = pairs ? 2 * kTcBM : kTcBM, at_once = pairs ? num_sms() / 2 : num_sms();
    const long tiles = (M + rows - 1) / rows * ((columns + kTcBN - 1) / kTcBN), waves = (tiles + at_once - 1) / at_once;
    const double full = (double)tiles / at_once;
    const double slice = waves > 1 ? (pairs ? 0.37 : 0.40) : pairs ? 0.285 + 0.055 * full : 0.335 + 0.045 * full;
    return 8.0 + std::max((double)columns * K * 2 / 6.2e6, waves * slices * slice);
}
static bool takes_pairs(int M, int N, int K, bool dual)
{
    return M > kTcBM && persistent_us(M, N, K, dual, true) < persistent_us(M, N, K, dual, false);
}

// The plan with the least estimated time in us, from a sweep on B200 over 70 to 1000 tokens of the 2048- and 4096-wide shapes
// (the estimate is within 15 % of all but the largest).  Either kernel needs about 8 us around its slices of 64 k.  A slice here takes 0.32 us, 0.45 when two blocks
// share an SM; the operands of all blocks come in at no more than 15 TB/s, the weights at 6.2.  Clusters of more than two blocks leave some
// slots of two blocks an SM unused (1030 tokens, 2048 outputs, K 5632, 288 blocks: clusters of two 28.1 us, the persistent kernel 37.0), and a
// second wave of blocks costs another start.
static SplitPlan plan_split(int M, int N, int K, bool dual, bool pairs)
{
    const int slices = (K + kTcBK - 1) / kTcBK, tiles_m = (M + kTcBM - 1) / kTcBM, columns = dual ? 2 * N : N;
    SplitPlan plan = {0, slices};
    const long tiles = (long)tiles_m * ((columns + kSplitBN - 1) / kSplitBN);
    const long sms = num_sms();
    if (tiles > 5 * sms) return plan;
    const double weights = (double)columns * K * 2 / 6.2e6;
    double best = persistent_us(M, N, K, dual, takes_pairs(M, N, K, dual));
    for (int ks = 1; ks <= (pairs ? 4 : 8); ks++) {
        const int per = (slices + ks - 1) / ks;
        if (ks > 1 && (per < 2 || per * (ks - 1) >= slices)) continue;  // every rank has slices
        const long blocks = tiles * ks, slots = ks <= 2 && !pairs ? 2 * sms : 2 * sms - 32;
        const long full = blocks / slots, rest = blocks % slots;
        const double time = full * per * 0.45 + (rest > sms ? per * 0.45 : rest ? per * 0.32 : 0.0);
        const double operands = (double)tiles * slices * kSplitStage / 15e6;
        const double t = 7.5 + 0.15 * ks + std::max({time, operands, weights}) + 6.0 * (full + (rest > 0) - 1);
        if (t < (plan.ks == 0 ? best - 1.0 : 0.97 * best)) {
            best = t;
            plan = {ks, per};
        }
    }
    return plan;
}

// Blocks of the launch's kernel that are sure to run at once in clusters of `size`, asked once per device.  The calculator answers one block
// per SM for a kernel with tensor memory; two fit.
template <typename Kern>
static int split_places(Kern kern, const cudaLaunchConfig_t& cfg, int size)
{
    static std::mutex mu;
    static std::map<std::tuple<const void*, int, int>, int> known;  // the kernels share their type
    std::lock_guard<std::mutex> lock(mu);
    int& n = known[std::make_tuple((const void*)kern, size, current_device())];
    if (n == 0) {
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) != cudaSuccess || clusters < 1) {
            (void)cudaGetLastError();
            clusters = num_sms() / size;
        }
        n = 2 * clusters * size;
    }
    return n;
}

template <typename T, int MODE>
static cudaError_t launch_split(const CUtensorMap& a, const CUtensorMap& b, const CUtensorMap& b2, T* y, int M, int N, int K, const TcEpilogue& epi,
                                const SplitPlan& plan, cudaStream_t st)
{
    auto kern = gemm_tc_split_kernel<T, MODE>;
    static DeviceOnce attr;
    const cudaError_t e = attr.run([kern] {
        const cudaError_t r = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSplitSmem);
        return r != cudaSuccess ? r : prefer_max_shared((const void*)kern);
    });
    if (e != cudaSuccess) return e;
    constexpr int kOutN = MODE == 2 ? kSplitBN / 2 : kSplitBN;
    const bool pairs = epi.ss_out != nullptr;
    int tiles_n = (N + kOutN - 1) / kOutN;
    if (pairs) tiles_n = (tiles_n + 1) & ~1;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = pairs ? 2 : 1;
    at[0].val.clusterDim.y = plan.ks;
    at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3(tiles_n * ((M + kTcBM - 1) / kTcBM), plan.ks, 1);
    cfg.blockDim = dim3(kSplitThreads);
    cfg.dynamicSmemBytes = kSplitSmem;
    cfg.stream = st;
    cfg.attrs = at;
    // Clusters that only just fit beside each other wait for the end of the kernel in front: started beside its last blocks they take places of a
    // GPC such that the last of them find no room for all their blocks until others are through (129 to 256 tokens, 4096 outputs, 32 clusters of
    // eight where 30 are sure to fit: every second projection took 29 instead of 19, 52 instead of 33 us).  All others start early.  Four layers
    // of 4096 (2048, 5120), us, all behind the end | as here: 130 tokens 781 | 781 (475 | 461, 947 | 928), 66 tokens 719 | 687 (460 | 433, 892 | 889).
    const int size = at[0].val.clusterDim.x * at[0].val.clusterDim.y;
    cfg.numAttrs = 1;
    if (size <= 2 || (int)(cfg.gridDim.x * cfg.gridDim.y) <= split_places(kern, cfg, size)) cfg.numAttrs = 2;
    note_launch();
    return cudaLaunchKernelEx(&cfg, kern, a, b, b2, y, M, N, K, epi, tiles_n, plan.per);
}

template <typename T, int MODE>
static cudaError_t launch_pairs(const CUtensorMap& a, const CUtensorMap& b, const CUtensorMap& b2, T* y, int M, int N, int K, const TcEpilogue& epi,
                                cudaStream_t st)
{
    auto kern = gemm_tc_kernel<T, MODE, false, true>;
    static DeviceOnce attr;
    const cudaError_t e = attr.run([kern] {
        const cudaError_t r = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcSmemBytes);
        return r != cudaSuccess ? r : prefer_max_shared((const void*)kern);
    });
    if (e != cudaSuccess) return e;
    constexpr int kOutN = MODE == 2 ? kTcBN / 2 : kTcBN;
    const long tiles = (long)((N + kOutN - 1) / kOutN) * ((M + 2 * kTcBM - 1) / (2 * kTcBM));
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3(2 * (unsigned)std::min<long>(tiles, num_sms() / 2));
    cfg.blockDim = dim3(kTcThreads);
    cfg.dynamicSmemBytes = kTcSmemBytes;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    note_launch();
    return cudaLaunchKernelEx(&cfg, kern, a, b, b2, y, M, N, K, epi, RowGroups{});
}

// mode 0: W [K,N]; 1: W [N,K]; 2: W and W2 [K,N], y = silu(x.W) * (x.W2)
template <typename T>
static int gemm_tc_launch(const T* x, const T* W, const T* W2, T* y, int M, int N, int K, int mode, cudaStream_t st,
                          const TcEpilogue& epi = TcEpilogue{})
{
    ONELLM_REQUIRE(K % 8 == 0 && N % 8 == 0, ONELLM_ERR_UNSUPPORTED, "gemm: M > 64 needs K %% 8 == 0 and N %% 8 == 0 (K=%d N=%d)",
                   K, N);
    CUtensorMap map_a, map_b, map_b2;
    int rc = make_map(&map_a, x, (uint64_t)K, (uint64_t)M, kTcBM);
    if (rc) return rc;
    rc = mode == 1 ? make_map(&map_b, W, (uint64_t)K, (uint64_t)N, kTcBN) : make_map(&map_b, W, (uint64_t)N, (uint64_t)K, kTcBK);
    if (rc) return rc;
    map_b2 = map_b;
    if (mode == 2) {
        rc = make_map(&map_b2, W2, (uint64_t)N, (uint64_t)K, kTcBK);
        if (rc) return rc;
    }
    const SplitPlan plan = plan_split(M, N, K, mode == 2, epi.ss_out != nullptr);
    if (plan.ks > 0) {
        if (mode == 1) RC(make_map(&map_b, W, (uint64_t)K, (uint64_t)N, kSplitBN));
        ONELLM_CUDA(mode == 0   ? (launch_split<T, 0>(map_a, map_b, map_b2, y, M, N, K, epi, plan, st))
                    : mode == 1 ? (launch_split<T, 1>(map_a, map_b, map_b2, y, M, N, K, epi, plan, st))
                                : (launch_split<T, 2>(map_a, map_b, map_b2, y, M, N, K, epi, plan, st)));
        return ONELLM_OK;
    }
    if (takes_pairs(M, N, K, mode == 2)) {
        if (mode == 1) RC(make_map(&map_b, W, (uint64_t)K, (uint64_t)N, kTcBN / 2));
        ONELLM_CUDA(mode == 0   ? (launch_pairs<T, 0>(map_a, map_b, map_b2, y, M, N, K, epi, st))
                    : mode == 1 ? (launch_pairs<T, 1>(map_a, map_b, map_b2, y, M, N, K, epi, st))
                                : (launch_pairs<T, 2>(map_a, map_b, map_b2, y, M, N, K, epi, st)));
        return ONELLM_OK;
    }
    static DeviceOnce smem_attr[3];
    {
        const void* fn = mode == 0 ? (const void*)gemm_tc_kernel<T, 0> : mode == 1 ? (const void*)gemm_tc_kernel<T, 1> : (const void*)gemm_tc_kernel<T, 2>;
        ONELLM_CUDA(smem_attr[mode].run([fn] { return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcSmemBytes); }));
    }
    const int out_n = mode == 2 ? kTcBN / 2 : kTcBN;
    const long tiles = (long)((N + out_n - 1) / out_n) * ((M + kTcBM - 1) / kTcBM);
    ONELLM_REQUIRE(tiles <= 0x7fffffffL, ONELLM_ERR_UNSUPPORTED, "gemm: too many tiles");
    const dim3 grid((unsigned)std::min<long>(tiles, num_sms()));  // persistent: one block per SM (shared memory allows no more)
    if (mode == 0)
        ONELLM_CUDA(launch_pdl(gemm_tc_kernel<T, 0>, grid, dim3(kTcThreads), kTcSmemBytes, st, map_a, map_b, map_b2, y, M, N, K, epi, RowGroups{}));
    else if (mode == 1)
        ONELLM_CUDA(launch_pdl(gemm_tc_kernel<T, 1>, grid, dim3(kTcThreads), kTcSmemBytes, st, map_a, map_b, map_b2, y, M, N, K, epi, RowGroups{}));
    else
        ONELLM_CUDA(launch_pdl(gemm_tc_kernel<T, 2>, grid, dim3(kTcThreads), kTcSmemBytes, st, map_a, map_b, map_b2, y, M, N, K, epi, RowGroups{}));
    return ONELLM_OK;
}

// Row groups (bfloat16): x has g.rows rows in group order, the weights are stacked.
static int gemm_tc_grouped(const onellm_projection& p, const TcEpilogue& epi, cudaStream_t st)
{
    typedef __nv_bfloat16 T;
    const RowGroups& g = *p.groups;
    ONELLM_REQUIRE(g.off && g.tile_group && g.tile_row && g.n_tiles && g.max_tiles > 0 && g.rows > 0 && g.weights > 0 && !g.x_rows && !g.x_stride &&
                       !g.y_stride && g.w_stride == (long)p.K * p.N && !p.ldw && !p.ldx && !p.resid,
                   ONELLM_ERR_UNSUPPORTED, "project: more than 64 rows per group need a tile table, rows in group order and stacked weights");
    CUtensorMap map_a, map_b, map_b2;
    int rc = make_map(&map_a, p.x, (uint64_t)p.K, (uint64_t)g.rows, kTcBM);
    if (!rc) rc = make_map(&map_b, p.W, (uint64_t)p.N, (uint64_t)p.K * g.weights, kTcBK);
    map_b2 = map_b;
    if (!rc && p.W2) rc = make_map(&map_b2, p.W2, (uint64_t)p.N, (uint64_t)p.K * g.weights, kTcBK);
    if (rc) return rc;
    const void* fn = p.W2 ? (const void*)gemm_tc_kernel<T, 2, true> : (const void*)gemm_tc_kernel<T, 0, true>;
    static DeviceOnce attr[2];
    ONELLM_CUDA(attr[p.W2 ? 1 : 0].run([fn] { return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcSmemBytes); }));
    const int out_n = p.W2 ? kTcBN / 2 : kTcBN;
    const long tiles = (long)((p.N + out_n - 1) / out_n) * g.max_tiles;
    ONELLM_REQUIRE(tiles <= 0x7fffffffL, ONELLM_ERR_UNSUPPORTED, "gemm: too many tiles");
    const dim3 grid((unsigned)std::min<long>(tiles, num_sms()));
    if (p.W2)
        ONELLM_CUDA(launch_pdl(gemm_tc_kernel<T, 2, true>, grid, dim3(kTcThreads), kTcSmemBytes, st, map_a, map_b, map_b2, (T*)p.y, p.M, p.N, p.K, epi, g));
    else
        ONELLM_CUDA(launch_pdl(gemm_tc_kernel<T, 0, true>, grid, dim3(kTcThreads), kTcSmemBytes, st, map_a, map_b, map_b2, (T*)p.y, p.M, p.N, p.K, epi, g));
    return ONELLM_OK;
}

int gemm_f16_large(const __half* x, const __half* W, __half* y, int M, int N, int K, int w_layout, cudaStream_t st)
{
    return gemm_tc_launch<__half>(x, W, nullptr, y, M, N, K, w_layout == ONELLM_W_NK ? 1 : 0, st);
}

// Gate and up projections with SwiGLU in the epilogue, M > 64.
int gemm_swiglu_f16_large(const __half* x, const __half* Wg, const __half* Wu, __half* out, int M, int I, int K, cudaStream_t st)
{
    return gemm_tc_launch<__half>(x, Wg, Wu, out, M, I, K, 2, st);
}

// Column tiles of a projection with N outputs (two weights: gate and up share a tile): the second extent of the
// [M, parts] array of partial row sums that onellm_gemm_rows writes.
int gemm_rows_parts(int N, bool dual)
{
    const int out_n = dual ? kTcBN / 2 : kTcBN;
    return (N + out_n - 1) / out_n;
}

// The large-M form of the norm-free projections (see TcEpilogue).
int gemm_rows_f16(const __half* x, const __half* W, const __half* W2, __half* y, int M, int N, int K, const float* row_ss, int ss_parts,
                  float eps, const __half* resid, const __half* bias, float* ss_out, cudaStream_t st)
{
    TcEpilogue epi = {};
    epi.row_ss = row_ss;
    epi.ss_parts = ss_parts;
    epi.eps = eps;
    epi.resid = resid;
    epi.bias = resid ? bias : nullptr;
    epi.ss_out = ss_out;
    return gemm_tc_launch<__half>(x, W, W2, y, M, N, K, W2 ? 2 : 0, st, epi);
}

// The bfloat16 form (more than 64 tokens, or rows in one group) behind project().
int gemm_bf16_large(const onellm_projection& p, cudaStream_t st)
{
    typedef __nv_bfloat16 bf16;
    TcEpilogue epi = {};
    epi.resid = p.resid;
    epi.act = p.act;
    epi.limit = p.limit;
    epi.scale = p.scale;
    epi.ldy = p.ldy;
    epi.f32 = p.f32;
    if (p.groups) return gemm_tc_grouped(p, epi, st);
    return gemm_tc_launch<bf16>((const bf16*)p.x, (const bf16*)p.W, (const bf16*)p.W2, static_cast<bf16*>(p.y), p.M, p.N, p.K, p.W2 ? 2 : 0, st, epi);
}

static const TimeoutFlag timeout_flag(tc_flag_read_clear, tc_flag_address);

}  // namespace onellm
