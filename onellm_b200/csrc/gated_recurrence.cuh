// What the two forms of the gated recurrence's context pass share: the token by token one and the decode step
// (gated_recurrence.cu), and the one in chunks of tokens on the tensor cores (gated_recurrence_tc.cu).
#pragma once
#include "mixers.h"
#include "tc_common.cuh"

namespace onellm {

// sigmoid(x) and 1 - sigmoid(x), both with full relative precision; the fast exponential and division where the
// projections are bfloat16 (their error is far below the rounding of x)
template <typename T>
__device__ __forceinline__ void sigmoid_pair(float x, float& s, float& c)
{
    float e, r;
    if constexpr (sizeof(T) == 2) {
        e = __expf(-fabsf(x));
        r = __fdividef(1.f, 1.f + e);
    } else {
        e = expf(-fabsf(x));
        r = 1.f / (1.f + e);
    }
    s = x >= 0.f ? r : e * r;
    c = x >= 0.f ? e * r : r;
}
template <typename T>
__device__ __forceinline__ float silu_of(float x)
{
    float s, c;
    sigmoid_pair<T>(x, s, c);
    return x * s;
}
// 1 - f and silu(q) of one channel
template <typename T>
__device__ __forceinline__ void gate(float q, float z, float zb, float lower, float& g, float& qs)
{
    float s, c;
    sigmoid_pair<T>(z + zb, s, c);
    g = (1.f - lower) * c;
    sigmoid_pair<T>(q, s, c);
    qs = q * s;
}

// sigmoid(z) ^ inv_tau - 1 from the logarithm of the sigmoid
__device__ __forceinline__ float decay(float z, float inv_tau) { return expm1f(inv_tau * (fminf(z, 0.f) - log1pf(expf(-fabsf(z))))); }

struct GrParams {
    GatedRecurrence g;
    TokenPositions tp;
    int settled;  // see gated_recurrence (mixers.h)
};

template <typename T>
__device__ __forceinline__ void gr_load4(const T* src, float (&f)[4])
{
    if constexpr (sizeof(T) == 4) {
        const float4 x = *reinterpret_cast<const float4*>(src);
        f[0] = x.x; f[1] = x.y; f[2] = x.z; f[3] = x.w;
    } else {
        const uint2 x = *reinterpret_cast<const uint2*>(src);
        const float2 a = unpack2<T>(x.x), b = unpack2<T>(x.y);
        f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y;
    }
}

// Context passes in chunks (gated_recurrence_tc.cu): the calls it takes, its work space and the pass itself.
bool gr_chunked_takes(const GatedRecurrence& g, const TokenPositions& tp, int B, int tokens);
size_t gr_chunked_workspace(int tokens, int H, int dk, int dv);
int gr_chunked(const GrParams& p, int B, int tokens, cudaStream_t st);

}  // namespace onellm
