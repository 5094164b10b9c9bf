// float32 projections: the kernels for few tokens (gemm_f32.cu) and for many (gemm_f32_tc.cu) and their arguments.
#pragma once
#include "common.cuh"

namespace onellm {

// y[M,N] = x[M,K] . W, W [K,N] or (w_nk) [N,K], rows ldx, ldw, ldy apart; resid (rows ldy apart, may be y): resid + scale * result;
// gate >= 0: y holds the gate product of a gated pair and becomes gate_pair(y, result)
struct GemmF32 {
    const float *x, *W;
    float* y;
    int M, N, K;
    long ldx, ldw, ldy;
    bool w_nk;
    const float* resid;
    float scale;
    int gate;
    float limit;
};

constexpr int kF32SkinnyTokens = 64;
constexpr int kF32SkinnyK = 96;  // below, a warp of gemm_f32_skinny has no or few rows for all its lanes: the tiled kernel is as fast or faster
// Sizes, strides and alignment that gemm_f32_skinny covers: 16-byte rows.
bool gemm_f32_skinny_takes(const GemmF32& a);
cudaError_t gemm_f32_skinny(const GemmF32& a, cudaStream_t st);
bool gemm_f32_tc_takes(const GemmF32& a);
cudaError_t gemm_f32_tc(const GemmF32& a, cudaStream_t st);

}  // namespace onellm
