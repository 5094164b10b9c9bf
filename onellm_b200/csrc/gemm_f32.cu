// Projections of float32 callers (the reference's own type) for few tokens: the weight is streamed, once for every 16 tokens.
//
// Replaces the cuBLAS SGEMM behind launchLinearGemm (src/kernels/qkv_linear.cu:8-65 of the reference) for decode steps:
// y[M,N] = x[M,K] . W with M of a few rows is bound by the bytes of W, so what matters is how many of them are on their way.
// The tiled kernel (sgemm_kernel, skinny_gemm.cu) gives 64 x 64 outputs to a block whatever M is: 64 blocks for 4096 columns,
// 16 rows of W in flight, 0.06 TB/s.  Here a thread keeps M x 4 sums in registers and nothing goes through shared memory until
// the end:
//   W [K,N]  a warp covers 128 columns (16 bytes a lane) and takes every eighth group of kRows rows of its block's K range; the
//            rows of the next group are requested before the sums of the current one; x is read by all lanes from the same
//            address (L1).  K is split over the eight warps of a block and over the blocks of a cluster; the partial sums meet
//            in shared memory, warps first, then ranks, both in a fixed order.
//   W [N,K]  a warp takes 4 rows of W and runs along K, 16 bytes a lane, so that W and x are read alike; sums over the lanes
//            by shuffles at the end, over the warps that share a row group through shared memory.
// Sums of products are in float throughout, in more and shorter chains than the tiled kernel's (error against 64 bits of a layer
// and the head: 5.9e-7 instead of 2.7e-6).
// Measured, 2 tokens, one 7B-shaped layer and its head (1.33 GB of weights, floor 0.20 ms): 6.65 ms in the tiled kernel, 0.33 here.
// 4096 x 12288 (201 MB), us, [K,N] | [N,K] | tiled: 2 tokens 48 | 44 | 893, 16 tokens 247 | 109 | 937, 32 tokens 470 | 197 | 1014,
// 64 tokens 935 | 361 | 1140.
#include <cooperative_groups.h>

#include <algorithm>

#include "gemm_f32.h"

namespace cg = cooperative_groups;

namespace onellm {

constexpr int kF32Threads = 256;
constexpr int kF32Warps = kF32Threads / 32;
constexpr int kF32Cols = 128;  // columns of a block, [K,N] form

__device__ __forceinline__ float4 ld_stream4(const float* p)
{
    const uint4 v = ld_nc_16(p);
    return make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w));
}

// x comes from the kernel in front of this one: a load that stays behind the dependency wait (a read-only one, __ldg, the
// compiler may move in front of it)
__device__ __forceinline__ float4 ld_dependent4(const float* p)
{
    float4 v;
    asm volatile("ld.global.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void store_f32(const GemmF32& a, int m, int n, float v)
{
    const size_t at = (size_t)m * a.ldy + n;
    if (a.resid) v = fmaf(v, a.scale, a.resid[at]);
    if (a.gate >= 0) v = gate_pair<true>(a.y[at], v, a.gate, a.limit);
    a.y[at] = v;
}

// grid (ceil(N / 128), KS, ceil(M / MT)), cluster (1, KS, 1); rows_per_block: a multiple of kRows
template <int MT, int kRows>
__global__ void __launch_bounds__(kF32Threads, 2)
gemv_kn_f32_kernel(const GemmF32 a, int rows_per_block)
{
    extern __shared__ __align__(16) float red[];  // [warps][MT][128]
    cg::cluster_group cluster = cg::this_cluster();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.z * MT, m_rows = min(MT, a.M - m0);
    const int n0 = blockIdx.x * kF32Cols, col = n0 + 4 * lane;
    const bool col_ok = col < a.N;  // N is a multiple of 4
    const int k_begin = blockIdx.y * rows_per_block, k_end = min(k_begin + rows_per_block, a.K);
    const float* w = a.W + (col_ok ? col : 0);
    const float* x = a.x + (size_t)m0 * a.ldx;

    float acc[MT][4];
#pragma unroll
    for (int m = 0; m < MT; m++)
#pragma unroll
        for (int c = 0; c < 4; c++) acc[m][c] = 0.f;
    float4 cur[kRows];
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    auto fetch = [&](int k, float4 (&v)[kRows]) {
#pragma unroll
        for (int r = 0; r < kRows; r++) v[r] = col_ok && k + r < k_end ? ld_stream4(w + (size_t)(k + r) * a.ldw) : zero;
    };
    pdl_wait();
    int k = k_begin + warp * kRows;
    fetch(k, cur);
    for (; k < k_end; k += kF32Warps * kRows) {
        float4 next[kRows];
        fetch(k + kF32Warps * kRows, next);
#pragma unroll
        for (int r4 = 0; r4 < kRows; r4 += 4) {
            const bool in = k + r4 < k_end;  // K and the rows of a block are multiples of 4
#pragma unroll
            for (int m = 0; m < MT; m++) {
                const float4 xv = in ? ld_dependent4(x + (size_t)min(m, m_rows - 1) * a.ldx + k + r4) : zero;
                const float xs[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    acc[m][0] = fmaf(xs[r], cur[r4 + r].x, acc[m][0]);
                    acc[m][1] = fmaf(xs[r], cur[r4 + r].y, acc[m][1]);
                    acc[m][2] = fmaf(xs[r], cur[r4 + r].z, acc[m][2]);
                    acc[m][3] = fmaf(xs[r], cur[r4 + r].w, acc[m][3]);
                }
            }
        }
#pragma unroll
        for (int r = 0; r < kRows; r++) cur[r] = next[r];
    }
    pdl_launch_dependents();
    float4* red4 = reinterpret_cast<float4*>(red);
#pragma unroll
    for (int m = 0; m < MT; m++) red4[(warp * MT + m) * 32 + lane] = make_float4(acc[m][0], acc[m][1], acc[m][2], acc[m][3]);
    __syncthreads();
    // the warps of a block, in order, into the first slice
    for (int e = tid; e < MT * 32; e += kF32Threads) {
        float4 s = red4[e];
#pragma unroll
        for (int v = 1; v < kF32Warps; v++) {
            const float4 p = red4[v * MT * 32 + e];
            s.x += p.x;
            s.y += p.y;
            s.z += p.z;
            s.w += p.w;
        }
        red4[e] = s;
    }
    cluster.sync();
    // the blocks of the cluster, in rank order; a rank finishes every KS-th output
    const int ks = gridDim.y, rank = blockIdx.y;
    for (int e = rank * kF32Threads + tid; e < MT * kF32Cols; e += ks * kF32Threads) {
        float p[8];
#pragma unroll
        for (int r = 0; r < 8; r++) p[r] = r < ks ? cluster.map_shared_rank(red, r)[e] : 0.f;
        float s = p[0];
#pragma unroll
        for (int r = 1; r < 8; r++) s += p[r];
        const int m = e / kF32Cols, n = n0 + e % kF32Cols;
        if (m < m_rows && n < a.N) store_f32(a, m0 + m, n, s);
    }
    cluster.sync();  // peers may still be reading this block's sums
}

// Warps of a block: kF32Warps / wk row groups of 4 rows, each shared by wk warps that take every wk-th 128 columns.
template <int MT>
__global__ void __launch_bounds__(kF32Threads, MT > 8 ? 1 : 2)
gemv_nk_f32_kernel(const GemmF32 a, int wk)
{
    __shared__ float red[kF32Warps][4 * MT];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.z * MT, m_rows = min(MT, a.M - m0);
    const int group = warp / wk, part = warp % wk;
    const int n0 = (blockIdx.x * (kF32Warps / wk) + group) * 4;
    const float* x = a.x + (size_t)m0 * a.ldx;
    const float* w[4];
#pragma unroll
    for (int r = 0; r < 4; r++) w[r] = a.W + (size_t)min(n0 + r, a.N - 1) * a.ldw;
    float acc[4][MT];
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
        for (int m = 0; m < MT; m++) acc[r][m] = 0.f;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    pdl_wait();
    if (n0 < a.N) {
        float4 cur[4];
        int k = part * 128 + 4 * lane;
        auto fetch = [&](int at, float4 (&v)[4]) {
#pragma unroll
            for (int r = 0; r < 4; r++) v[r] = at < a.K ? ld_stream4(w[r] + at) : zero;  // K is a multiple of 4
        };
        fetch(k, cur);
        for (; k - 4 * lane < a.K; k += wk * 128) {
            float4 next[4];
            fetch(k + wk * 128, next);
#pragma unroll
            for (int m = 0; m < MT; m++) {
                const float4 xv = k < a.K ? ld_dependent4(x + (size_t)min(m, m_rows - 1) * a.ldx + k) : zero;
#pragma unroll
                for (int r = 0; r < 4; r++)
                    acc[r][m] = fmaf(xv.x, cur[r].x, fmaf(xv.y, cur[r].y, fmaf(xv.z, cur[r].z, fmaf(xv.w, cur[r].w, acc[r][m]))));
            }
#pragma unroll
            for (int r = 0; r < 4; r++) cur[r] = next[r];
        }
    }
    pdl_launch_dependents();
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
        for (int m = 0; m < MT; m++) {
            const float s = warp_sum(acc[r][m]);
            if (lane == 0) red[warp][m * 4 + r] = s;
        }
    __syncthreads();
    for (int e = tid; e < (kF32Warps / wk) * 4 * MT; e += kF32Threads) {
        const int g = e / (4 * MT), i = e % (4 * MT), m = i / 4;
        const int n = (blockIdx.x * (kF32Warps / wk) + g) * 4 + i % 4;
        float s = red[g * wk][i];
        for (int p = 1; p < wk; p++) s += red[g * wk + p][i];
        if (m < m_rows && n < a.N) store_f32(a, m0 + m, n, s);
    }
}

template <int MT, int kRows>
static cudaError_t launch_kn(const GemmF32& a, cudaStream_t st)
{
    auto kern = gemv_kn_f32_kernel<MT, kRows>;
    constexpr size_t smem = (size_t)kF32Warps * MT * kF32Cols * sizeof(float);
    static DeviceOnce attr;
    const cudaError_t e = attr.run([kern] {
        const cudaError_t r = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        return r != cudaSuccess ? r : prefer_max_shared((const void*)kern);
    });
    if (e != cudaSuccess) return e;
    // K split (= cluster size): as many blocks as fill the GPU twice, of at least two groups of rows for every warp
    const int cols = (a.N + kF32Cols - 1) / kF32Cols, z = (a.M + MT - 1) / MT;
    int ks = 1;
    while (ks < 8 && (long)cols * z * ks < 2L * num_sms() && a.K >= 2 * (ks + 1) * kF32Warps * kRows) ks++;
    const int unit = kRows;
    const int per = ((a.K + ks - 1) / ks + unit - 1) / unit * unit;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 1;
    at[0].val.clusterDim.y = ks;
    at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3(cols, ks, z);
    cfg.blockDim = dim3(kF32Threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    note_launch();
    return cudaLaunchKernelEx(&cfg, kern, a, per);
}

template <int MT>
static cudaError_t launch_nk(const GemmF32& a, cudaStream_t st)
{
    const int z = (a.M + MT - 1) / MT;
    int wk = 1;
    while (wk < kF32Warps && (long)((a.N + 31) / 32) * wk * z < 4L * num_sms() && a.K >= 512 * wk) wk *= 2;
    const int rows = 4 * (kF32Warps / wk);
    return launch_pdl(gemv_nk_f32_kernel<MT>, dim3((a.N + rows - 1) / rows, 1, z), dim3(kF32Threads), 0, st, a, wk);
}

bool gemm_f32_skinny_takes(const GemmF32& a)
{
    return a.M <= kF32SkinnyTokens && a.K >= kF32SkinnyK && a.K % 4 == 0 && a.ldx % 4 == 0 && a.ldw % 4 == 0 && (a.w_nk || a.N % 4 == 0) && aligned16(a.x) && aligned16(a.W);
}

cudaError_t gemm_f32_skinny(const GemmF32& a, cudaStream_t st)
{
    if (a.w_nk) {
        if (a.M <= 1) return launch_nk<1>(a, st);
        if (a.M <= 2) return launch_nk<2>(a, st);
        if (a.M <= 4) return launch_nk<4>(a, st);
        if (a.M <= 8) return launch_nk<8>(a, st);
        return launch_nk<16>(a, st);
    }
    if (a.M <= 1) return launch_kn<1, 8>(a, st);
    if (a.M <= 2) return launch_kn<2, 8>(a, st);
    if (a.M <= 4) return launch_kn<4, 8>(a, st);
    if (a.M <= 8) return launch_kn<8, 8>(a, st);
    return launch_kn<16, 4>(a, st);
}

}  // namespace onellm
