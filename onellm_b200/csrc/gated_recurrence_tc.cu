// Gated outer-product recurrences over long prompts (bfloat16 projections): chunks of 128 tokens as products on the tensor cores, with
// the precision of float.
//
// Token by token a head's state goes through every multiply-add on the cores that hold it, one token after the other.  Over a chunk
// the recurrence is three products.  With d = 1 - f, b_t the product of the gates from the chunk's first token to t, and
// m the point between tokens 63 and 64:
//     q~_t = q_t b_t / b_m,  k~_j = k_j b_m / b_j                  (TIED: k = d)
//     o_t = (q~_t b_m)^T S + sum over j <= t of (q~_t . k~_j) v_j,   S <- b S + (b / b_m) k~^T V       (b: of the whole chunk)
// which is the chunk form of gated linear attention (Yang et al., "Gated Linear Attention Transformers with Hardware-Efficient
// Training", 2023).  Anchored in its middle, a chunk's factors stay in the range of float while half a chunk forgets no channel below 2^-80.
//
// Every operand is float: it is the sum of three bf16 values (see gemm_f32_tc.cu), values of the projections are bf16 themselves.  Of two
// such sums six products count (the others are below 2^-26 of the whole), of a sum and a value three.  The tensor cores truncate when they
// add, so the small products have an accumulator of their own, or go first, and the state's are cut every 32 tokens and added in registers.
// Gates are multiplied up with their rounding errors (1 - d is not a float), so that hundreds of equal gates stay exact.
//
// Three launches (us at 1 x 2000 tokens, 16 heads of 128 x 128, TIED | 2 x 1030 tokens, 4 heads of 256 x 512, KEYED):
//   1. gr_chunk_prepare_kernel (26 | 37): gates, their products outward from the middle of the chunk, the pieces of q~ and k~, a copy of the
//      values in whole chunks.  A channel that forgets too much has q b_t and k b / b_j instead.  Bound by the instructions (70 per
//      channel and token).
//   2. gr_chunk_state_kernel (29 | 24): a block keeps 32 or 64 key channels x 128 value columns of a state in registers and walks the
//      chunks; it leaves the pieces of b_m S in front of every chunk.  Bound by the chain of a chunk: products into registers, update, split.
//      Blocks behind these make the parts of the tables (q_t . k_j) that channels without quotients owe, see gd_table.
//   3. gr_chunk_output_kernel (26 | 58): a block makes 128 tokens x 128 value columns of the output: q~ . k~, q~ . S, then, behind the mask,
//      the first times V with the pieces of the table in tensor memory; RMS norm over the head (a cluster's blocks share the sums) and gate.
//      Bound by its operands: 6 bytes a float, 320 KB (608 KB) for 7680 (13800) cycles of products.
// All three 85 | 121 us; token by token 255 | 244.  With one channel a head that forgets too much 115 | 163, where the gates are sigmoids of
// normal numbers 181 | 202, where all channels do 239 | 234.  A short call with such channels is slower than token by token, which no rule
// on sizes can know: 1 x 288 tokens 38 | 57 us without, 59 | 81, 82 | 99 and 103 | 119 with them, token by token 42 | 73; 1 x 768 tokens TIED 48
// without, 73, 110 and 132, token by token 101.  Error of the state against 64 bits 9.7e-8 | 8.3e-8 (9.3e-8 | 1.1e-7; sigmoids of normal numbers
// 8.7e-8 | 6.3e-8, 7.0e-8 | 5.3e-8), of the outputs 1.66e-3 both, the rounding to bfloat16.
// A value that is not finite would reach the chunk's earlier tokens through a product with zero: the copy has zero there, and the
// column is NaN from its token on.
#include <cooperative_groups.h>

#include <algorithm>
#include <mutex>

#include "gated_recurrence.cuh"

namespace cg = cooperative_groups;

namespace onellm {

typedef __nv_bfloat16 bf16;

constexpr int kGcTok = 128;                        // tokens of a chunk
constexpr int kGcMaxDk = 256, kGcMaxDv = 1024, kGcMaxRank = 64;
constexpr int kGcTile = kGcTok * 64 * 2;           // bytes of 128 rows of 64 columns
constexpr float kGcLeast = 0x1p-80f, kGcMost = 0x1p20f;

// What the launches hand on, for chunk s of the pass's head h at index `at` = h * slots + s.  Operands lie as the tensor cores read them, in tiles of
// 128 rows x 64 columns (16 KB, 128-byte rows swizzled), so that one copy of contiguous bytes brings them in.
struct GrChunks {
    int slots;            // chunks of all sequences, at most
    int head0, heads;     // of this pass
    unsigned char *q, *k; // [dk / 64][3 pieces] tiles of tokens x channels
    unsigned char* s;     // [dv / 128][dk / 64][3 pieces] tiles of values x channels: b_m times the state in front of the chunk
    unsigned char* v;     // [dv / 64] tiles of tokens x values
    float* vec;           // [dk / 64][4][64]: b_m, b / b_m, and a, c of S <- a S + c S
    float* A;             // [128][128] a table by multiply-adds, where `notes` says so
    float* gate;          // [128][dk] 1 - f of the channels it has
    uint32_t* fast;       // [8] bits of these channels, there only where `notes` says so
    int* bad;             // [2][dv] first token of the chunk's half whose value is not finite, or 128; there only for a half that the notes name
    int4* notes;          // x: 1 A is the chunk's table, 2 A is added to it; y, z: the first, the second half of the tokens has values that are not finite;
                          // w: these values have been divided by 2 to the power of the low, the high half word
};
static size_t gc_chunk_bytes(int dk, int dv)
{
    return (size_t)2 * 3 * kGcTok * dk * 2 + (size_t)3 * dv * dk * 2 + (size_t)kGcTok * dv * 2 + (size_t)4 * dk * 4 + (size_t)kGcTok * kGcTok * 4 +
           (size_t)2 * dv * 4 + (size_t)4 * kGcTok * dk + 32 + 16;
}
__device__ __forceinline__ float two_to(int e) { return __int_as_float((127 + e) << 23); }
// place of an element in a tile
__device__ __forceinline__ uint32_t gc_at(int row, int col) { return (uint32_t)(row * 128 + (((col >> 3) ^ (row & 7)) << 4) + (col & 7) * 2); }

// Chunk `slot` counted over all sequences: its sequence and its place there; false behind the last one (every warp as a whole)
__device__ __forceinline__ bool gc_locate(const int* cu, int B, int slot, int& b, int& i)
{
    const int lane = threadIdx.x & 31;
    int base = 0;
    for (int b0 = 0; b0 < B; b0 += 32) {
        const int n = b0 + lane < B ? (cu[b0 + lane + 1] - cu[b0 + lane] + kGcTok - 1) / kGcTok : 0;
        int s = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += up;
        }
        const unsigned there = __ballot_sync(0xffffffffu, slot < base + s);
        if (there) {
            const int l = __ffs(there) - 1;
            b = b0 + l;
            i = slot - base - __shfl_sync(0xffffffffu, s - n, l);
            return true;
        }
        base += __shfl_sync(0xffffffffu, s, 31);
    }
    return false;
}

// chunks of all sequences (every warp as a whole)
__device__ __forceinline__ int gc_count(const int* cu, int B)
{
    int n = 0;
    for (int e = threadIdx.x & 31; e < B; e += 32) n += (cu[e + 1] - cu[e] + kGcTok - 1) / kGcTok;
    return __reduce_add_sync(0xffffffffu, n);
}

// Product of gates 1 - d as hi + lo: what rounding takes away (of 1 - d too, again and again the same for equal gates) is kept.
struct GateProduct {
    float hi = 1.f, lo = 0.f;
    __device__ __forceinline__ void times(float d)
    {
        const float f = 1.f - d, e = (1.f - f) - d, p = hi * f;
        lo = fmaf(lo, f, fmaf(hi, e, fmaf(hi, f, -p)));
        hi = p;
    }
    __device__ __forceinline__ void times(float h, float l)
    {
        const float p = hi * h;
        lo = fmaf(lo, h, fmaf(hi, l, fmaf(hi, h, -p)));
        hi = p;
    }
    __device__ __forceinline__ float value() const { return hi + lo; }
};
// 1 / x of a normal number: the approximate reciprocal and one Newton step
__device__ __forceinline__ float reciprocal(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return fmaf(r, fmaf(-x, r, 1.f), r);
}
// S <- alpha S + gamma S for a gate product: in the form that keeps the digits of one near 1
__device__ __forceinline__ void decay_form(const GateProduct& b, float& alpha, float& gamma)
{
    const bool near = b.hi > 0.5f;
    alpha = near ? (b.hi - 1.f) + b.lo : b.value();
    gamma = near ? 1.f : 0.f;
}

// 1 - f of a channel and token
template <bool KEYED>
__device__ __forceinline__ float gc_forget(const GatedRecurrence& p, float z, float zb, float lower)
{
    if constexpr (KEYED) return -decay(z, p.inv_tau);
    float s, c;
    sigmoid_pair<bf16>(z + zb, s, c);
    return (1.f - lower) * c;
}

__device__ __forceinline__ void gc_store_pieces(unsigned char* dst, float lo, float hi)
{
    uint32_t p0, p1, p2, rest = 0u;
    split_pair(lo, hi, p0, p1, p2, rest);
    *reinterpret_cast<uint32_t*>(dst) = p0;
    *reinterpret_cast<uint32_t*>(dst + kGcTile) = p1;
    *reinterpret_cast<uint32_t*>(dst + 2 * kGcTile) = p2;
}

// The values of half a chunk's tokens in tiles, zero behind its last token and where they are not finite.  Where any is kGcMost or more, all are
// divided by the power of two that brings them below: k~ is up to 2^80 times 2^20, and that times 2^20 and 64 tokens is all that float holds.
// (By halves of the tokens, each with a power of its own: a block with half the columns of all of them had to hear of the other half's, at 4 us
// of 82 by looking through that as well, 9 by a word of the other block.)
__device__ __forceinline__ void gc_values(const GatedRecurrence& p, const GrChunks& ck, size_t at, int h, int half, int t0, int n, int* s_bad, int* s_most)
{
    const int tid = threadIdx.x, dv = p.dv, groups = dv / 4, from = half * (kGcTok / 2);
    for (int e = tid; e < dv; e += blockDim.x) s_bad[e] = kGcTok;
    if (tid == 0) *s_most = 0;
    __syncthreads();
    const bf16* src = reinterpret_cast<const bf16*>(p.v) + (size_t)t0 * p.ld + (size_t)h * dv;
    unsigned char* dst = ck.v + at * (dv / 64) * kGcTile;
    auto place = [&](int e) { return reinterpret_cast<uint2*>(dst + (size_t)((e % groups) * 4 >> 6) * kGcTile + gc_at(from + e / groups, (e % groups) * 4 & 63)); };
    bool bad = false;
#pragma unroll 8
    for (int e = tid; e < kGcTok / 2 * groups; e += blockDim.x) {
        const int t = from + e / groups, col = (e % groups) * 4;
        uint2 x = make_uint2(0u, 0u);
        if (t < n) x = *reinterpret_cast<const uint2*>(src + (size_t)t * p.ld + col);
        // a value whose exponent's field reaches 147, kGcMost or more; all ones where it is not finite
        const uint32_t most = (((x.x & 0x7f807f80u) + 0x36803680u) | ((x.y & 0x7f807f80u) + 0x36803680u)) & 0x80008000u;
        if (most) {
            uint32_t w[2] = {x.x, x.y};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const uint32_t part = 0xffffu << (16 * (j & 1)), top = 0x7f80u << (16 * (j & 1));
                if ((w[j >> 1] & top) == top) {
                    w[j >> 1] &= ~part;
                    atomicMin(&s_bad[col + j], t);
                    bad = true;
                } else {
                    atomicMax(s_most, (int)((w[j >> 1] & top) >> (16 * (j & 1))));
                }
            }
            x = make_uint2(w[0], w[1]);
        }
        *place(e) = x;
    }
    const bool any = __syncthreads_or(bad);
    const int down = max((*s_most >> 7) - 146, 0);
    if (any)
        for (int e = tid; e < dv; e += blockDim.x) ck.bad[(at * 2 + half) * dv + e] = s_bad[e];
    if (down) {
        const float scale = two_to(-down);
        for (int e = tid; e < kGcTok / 2 * groups; e += blockDim.x) {  // what this thread has written
            const float2 a = unpack2<bf16>(place(e)->x), b = unpack2<bf16>(place(e)->y);
            *place(e) = make_uint2(pack2<bf16>(a.x * scale, a.y * scale), pack2<bf16>(b.x * scale, b.y * scale));
        }
    }
    if (tid == 0) {
        (half ? ck.notes[at].z : ck.notes[at].y) = any;
        reinterpret_cast<short*>(&ck.notes[at].w)[half] = (short)down;
    }
}

// Grid (slots, heads, 4), 2 dk threads, clusters of two.  z = 0 and 1 have the tokens in front of and behind the middle of the chunk: a thread two
// channels and a quarter of the tokens, in the order outward from the middle.  z = 2 and 3: the values.
// The loops are short on purpose: straight-line code is fetched once per block, by all SMs at the same time.
template <bool KEYED>
__global__ void __launch_bounds__(512, 2) gr_chunk_prepare_kernel(const __grid_constant__ GrParams pp, const __grid_constant__ GrChunks ck)
{
    constexpr int kSegs = 4, kHalf = kGcTok / 2, kSeg = kHalf / kSegs, kBatch = 4;
    const GatedRecurrence& p = pp.g;
    extern __shared__ __align__(16) float sm[];  // 1 - f [16][2 dk threads][2], the gate's low-rank input [64][rank]
    __shared__ float s_hi[kSegs][kGcMaxDk], s_lo[kSegs][kGcMaxDk], s_all[2][kGcMaxDk];
    __shared__ uint32_t s_fast[kGcMaxDk / 32];
    __shared__ int s_odd;  // 1: something is too large or not a number, 2: a channel forgets too much
    cg::cluster_group cluster = cg::this_cluster();
    pdl_wait();
    pdl_launch_dependents();
    int b, i;
    if (!gc_locate(pp.tp.cu, pp.tp.B, blockIdx.x, b, i)) return;  // the same in both blocks of a cluster
    const int tid = threadIdx.x, h = ck.head0 + blockIdx.y, dk = p.dk;
    const int t0 = pp.tp.cu[b] + i * kGcTok, n = min(kGcTok, pp.tp.cu[b + 1] - t0);
    const size_t at = (size_t)blockIdx.y * ck.slots + blockIdx.x;
    if (blockIdx.z >= 2) {
        gc_values(p, ck, at, h, blockIdx.z - 2, t0, n, reinterpret_cast<int*>(sm), &s_odd);
        return;
    }
    if (tid == 0) s_odd = 0;
    const bool back = blockIdx.z == 0;
    const int seg = tid / (dk / 2), c = (tid % (dk / 2)) * 2, hc = h * dk + c;
    const int first = back ? kHalf - 1 - seg * kSeg : kHalf + seg * kSeg, dir = back ? -1 : 1;
    const size_t row0 = (size_t)t0 * p.ld;
    float2* d = reinterpret_cast<float2*>(sm) + tid;  // this thread's: d[o * blockDim.x]
    const int D = blockDim.x;
    const float* s_r = sm + kHalf * dk;  // of token t at (t & 63)
    if constexpr (KEYED) {
        for (int e = tid; e < kHalf * p.rank; e += blockDim.x) {
            const int t = e / p.rank + (back ? 0 : kHalf);
            sm[kHalf * dk + e] = t < n ? to_float(reinterpret_cast<const bf16*>(p.r)[row0 + (size_t)t * p.ld + e % p.rank]) : 0.f;
        }
        __syncthreads();
    }
    const float2 zb = *reinterpret_cast<const float2*>(p.zb + hc);
    const float2 lower = KEYED ? make_float2(0.f, 0.f) : *reinterpret_cast<const float2*>(p.lower + hc);
    // gates that are none; a gate that is not a number shows in the products below
    bool odd = !KEYED && !(lower.x >= 0.f && lower.x <= 1.f && lower.y >= 0.f && lower.y <= 1.f);
    GateProduct b0, b1;
#pragma unroll 1
    for (int o0 = 0; o0 < kSeg; o0 += 8) {
        float2 z[8];
        if constexpr (KEYED) {
            const float *A0 = p.A + (size_t)hc * p.rank, *A1 = A0 + p.rank, *r0 = s_r + ((first + dir * o0) & (kHalf - 1)) * p.rank;
#pragma unroll
            for (int j = 0; j < 8; j++) z[j] = zb;
            int e = 0;
            if (p.rank % 4 == 0) {
                for (; e < p.rank; e += 4) {
                    const float4 a = *reinterpret_cast<const float4*>(A0 + e), w = *reinterpret_cast<const float4*>(A1 + e);
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        const float4 r = *reinterpret_cast<const float4*>(r0 + dir * j * p.rank + e);
                        z[j].x = fmaf(a.w, r.w, fmaf(a.z, r.z, fmaf(a.y, r.y, fmaf(a.x, r.x, z[j].x))));
                        z[j].y = fmaf(w.w, r.w, fmaf(w.z, r.z, fmaf(w.y, r.y, fmaf(w.x, r.x, z[j].y))));
                    }
                }
            }
            for (; e < p.rank; e++) {
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const float r = r0[dir * j * p.rank + e];
                    z[j].x = fmaf(A0[e], r, z[j].x);
                    z[j].y = fmaf(A1[e], r, z[j].y);
                }
            }
        } else {
            uint32_t w[8];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const int t = first + dir * (o0 + j);
                w[j] = t < n ? *reinterpret_cast<const uint32_t*>(reinterpret_cast<const bf16*>(p.z) + row0 + (size_t)t * p.ld + hc) : 0u;
            }
#pragma unroll
            for (int j = 0; j < 8; j++) z[j] = unpack2<bf16>(w[j]);
        }
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const bool in = first + dir * (o0 + j) < n;  // a token behind the last one keeps everything
            const float2 x = make_float2(in ? gc_forget<KEYED>(p, z[j].x, zb.x, lower.x) : 0.f, in ? gc_forget<KEYED>(p, z[j].y, zb.y, lower.y) : 0.f);
            b0.times(x.x);
            b1.times(x.y);
            d[(o0 + j) * D] = x;
        }
    }
    *reinterpret_cast<float2*>(&s_hi[seg][c]) = make_float2(b0.hi, b1.hi);
    *reinterpret_cast<float2*>(&s_lo[seg][c]) = make_float2(b0.lo, b1.lo);
    const bf16* qp = reinterpret_cast<const bf16*>(p.q) + row0 + hc;
    const bf16* kp = KEYED ? reinterpret_cast<const bf16*>(p.k) + row0 + hc : nullptr;
    uint32_t qr[kBatch];
    [[maybe_unused]] uint32_t kr[kBatch];
    auto fetch = [&](int o0) {
#pragma unroll
        for (int j = 0; j < kBatch; j++) {
            const int t = first + dir * (o0 + j);
            const bool in = o0 < kSeg && t < n;
            qr[j] = in ? *reinterpret_cast<const uint32_t*>(qp + (size_t)t * p.ld) : 0u;
            if constexpr (KEYED) kr[j] = in ? *reinterpret_cast<const uint32_t*>(kp + (size_t)t * p.ld) : 0u;
        }
    };
    fetch(0);
    __syncthreads();
    // the products of the parts between this one and the middle come first
    b0 = GateProduct(), b1 = GateProduct();
#pragma unroll 1
    for (int s = 0; s < seg; s++) {
        b0.times(s_hi[s][c], s_lo[s][c]);
        b1.times(s_hi[s][c + 1], s_lo[s][c + 1]);
    }
    const size_t tiles = (at * (dk / 64) + (c >> 6)) * 3 * kGcTile + (c & 7) * 2;
    unsigned char *q_dst = ck.q + tiles, *k_dst = ck.k + tiles;
    const int c16 = (c & 63) >> 3;
    __nv_bfloat162 most = __floats2bfloat162_rn(0.f, 0.f);  // of q and k in front of their factors, which are 2^80 at most
#pragma unroll 1
    for (int o0 = 0; o0 < kSeg; o0 += kBatch) {
        uint32_t qn[kBatch];
        [[maybe_unused]] uint32_t kn[kBatch];
#pragma unroll
        for (int j = 0; j < kBatch; j++) {
            qn[j] = qr[j];
            if constexpr (KEYED) kn[j] = kr[j];
        }
        fetch(o0 + kBatch);
#pragma unroll
        for (int j = 0; j < kBatch; j++) {
            const int t = first + dir * (o0 + j);
            const float2 x = d[(o0 + j) * D];
            float2 q = unpack2<bf16>(qn[j]), k = x;
            most = __hmax2(most, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&qn[j])));
            if constexpr (KEYED) {
                most = __hmax2(most, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&kn[j])));
                k = unpack2<bf16>(kn[j]);
                q.x *= p.q_scale, q.y *= p.q_scale;
            } else {
                q.x = silu_of<bf16>(q.x), q.y = silu_of<bf16>(q.y);
            }
            const GateProduct was0 = b0, was1 = b1;
            b0.times(x.x);
            b1.times(x.y);
            const float f0 = back ? was0.value() : b0.value(), f1 = back ? was1.value() : b1.value(), r0 = reciprocal(f0), r1 = reciprocal(f1);
            const uint32_t to = (uint32_t)(t * 128 + ((c16 ^ (t & 7)) << 4));
            gc_store_pieces(q_dst + to, q.x * (back ? r0 : f0), q.y * (back ? r1 : f1));
            gc_store_pieces(k_dst + to, k.x * (back ? f0 : r0), k.y * (back ? f1 : r1));
        }
    }
    bool less = false;
    odd |= !(__low2float(most) < kGcMost && __high2float(most) < kGcMost);
    if (KEYED) odd |= !(fabsf(p.q_scale) < kGcMost);
    if (seg == kSegs - 1) {  // these have come to the end of the chunk's half
        less = b0.hi < kGcLeast || b1.hi < kGcLeast;
        odd |= !(b0.hi >= 0.f && b1.hi >= 0.f);
        *reinterpret_cast<float2*>(&s_all[0][c]) = make_float2(b0.hi, b1.hi);
        *reinterpret_cast<float2*>(&s_all[1][c]) = make_float2(b0.lo, b1.lo);
    }
    if (odd || less) atomicOr(&s_odd, odd ? 1 : 2);
    cluster.sync();  // everything that either block has written
    const int notes = s_odd | *cluster.map_shared_rank(&s_odd, back ? 1 : 0);
    const float *back_hi = cluster.map_shared_rank(s_all[0], 0), *front_hi = cluster.map_shared_rank(s_all[0], 1);
    if (notes) {  // channels without quotients: see gd_table
        if (tid < dk) {
            const bool in = (notes & 1) || !(back_hi[tid] >= kGcLeast && front_hi[tid] >= kGcLeast);
            const uint32_t bits = __ballot_sync(0xffffffffu, in);
            if ((tid & 31) == 0) {
                s_fast[tid >> 5] = bits;
                if (back) ck.fast[at * 8 + (tid >> 5)] = bits;
            }
        }
        __syncthreads();
    }
    if (back) {
        const float* front_lo = cluster.map_shared_rank(s_all[1], 1);
        for (int e = tid; e < dk; e += blockDim.x) {
            GateProduct all;
            float* vec = ck.vec + at * 4 * dk + (e >> 6) * 256 + (e & 63);
            const bool plain = notes && (s_fast[e >> 5] >> (e & 31)) & 1u;
            all.times(s_all[0][e], s_all[1][e]);
            vec[0] = plain ? 1.f : all.value();
            vec[64] = plain ? 1.f : front_hi[e] + front_lo[e];
            all.times(front_hi[e], front_lo[e]);
            decay_form(all, vec[128], vec[192]);
        }
        if (tid == 0) ck.notes[at].x = notes & 1 ? 1 : notes;
    }
    const uint32_t mine = notes ? s_fast[c >> 5] >> (c & 31) & 3u : 0u;
    if (mine) {
        // q b_t and k b / b_j: one of them takes the gates between its token and the other half, and that half's, on the way out from the middle of
        // the chunk, the other one those on the far side of its token, on the way back.  The front half has q on the way out.
#pragma unroll 1
        for (int way = 0; way < 2; way++) {
            const bool out = way == 0, is_q = back != out;
            b0 = GateProduct(), b1 = GateProduct();
            if (out) {
                const float *hi = back ? front_hi : back_hi, *lo = cluster.map_shared_rank(s_all[1], back ? 1 : 0);
                b0.times(hi[c], lo[c]);
                b1.times(hi[c + 1], lo[c + 1]);
            }
#pragma unroll 1
            for (int s = out ? 0 : seg + 1; s < (out ? seg : kSegs); s++) {
                b0.times(s_hi[s][c], s_lo[s][c]);
                b1.times(s_hi[s][c + 1], s_lo[s][c + 1]);
            }
#pragma unroll 1
            for (int o0 = 0; o0 < kSeg; o0 += 8) {
                uint32_t w[8];
                if (is_q || KEYED) {
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        const int t = first + dir * (out ? o0 + j : kSeg - 1 - o0 - j);
                        w[j] = t < n ? *reinterpret_cast<const uint32_t*>((is_q ? qp : kp) + (size_t)t * p.ld) : 0u;
                    }
                }
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const int o = out ? o0 + j : kSeg - 1 - o0 - j, t = first + dir * o;
                    const float2 x = d[o * D];
                    float2 y = x;
                    if (is_q || KEYED) y = unpack2<bf16>(w[j]);
                    if (is_q) y = KEYED ? make_float2(y.x * p.q_scale, y.y * p.q_scale) : make_float2(silu_of<bf16>(y.x), silu_of<bf16>(y.y));
                    const float f0 = b0.value(), f1 = b1.value();
                    b0.times(x.x);
                    b1.times(x.y);
                    uint32_t piece[3], rest = 0u;
                    split_pair(y.x * (is_q ? b0.value() : f0), y.y * (is_q ? b1.value() : f1), piece[0], piece[1], piece[2], rest);
                    unsigned char* to = (is_q ? q_dst : k_dst) + (t * 128 + ((c16 ^ (t & 7)) << 4));
#pragma unroll
                    for (int e = 0; e < 3; e++) {
                        if (mine == 3u) *reinterpret_cast<uint32_t*>(to + e * kGcTile) = piece[e];
                        else *reinterpret_cast<unsigned short*>(to + e * kGcTile + (mine & 2u)) = (unsigned short)(mine == 1u ? piece[e] : piece[e] >> 16);
                    }
                    if (out) *reinterpret_cast<float2*>(ck.gate + (at * kGcTok + t) * dk + c) = x;
                }
            }
        }
    }
    cluster.sync();  // the other block may still be reading this one's products
}

// ---- 2. the states in front of the chunks --------------------------------------------------------------------
constexpr int kGsWarps = 16;
constexpr int kGsBlock = kGsWarps * 32 + 64;  // and one that issues the loads, one the products
constexpr int kGsHalf = kGcTile / 2;          // 64 tokens of a tile
constexpr int kGsStage = 5 * kGsHalf;         // of half a chunk: values 64 x 128, then three pieces of k~ 64 x 64
constexpr int kGsDepth = 4;
constexpr int kGsVec = 4 * 64 * 4;            // bytes of the chunk's vectors, four chunks in turn
constexpr int kGsSmem = kGsDepth * kGsStage + 3 * kGcTile + 4 * kGsVec;

__device__ __forceinline__ void gs_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kGsWarps * 32) : "memory"); }  // the warps that hold the state

// ---- channels without quotients
// A channel that forgets too much (below 2^-80 in half a chunk) has q b_t and k b / b_j in the place of q~ and k~, with the middle of the chunk at one.
// The table's product makes no more than 2^-80 of what is due of those, and the channel's own part of the table, by multiply-adds along the
// gates, is added to it.  Where q or k is too large or a gate is not a number, all channels of the chunk go that way and the sums
// here take the table's place.  The blocks behind those of the states make these parts of the table while those walk the chunks: several blocks to a
// chunk and head where there are few.  A warp has a strip of 8 tokens, its lanes the tokens in front: 32 at a time by what they are worth at the
// end of their 32, but for the strip's own 32, along the gates.  32 channels at a time, their values requested one group ahead.
constexpr int kGdGroup = 32, kGdRow = kGcTok + 4;
static_assert(6 * kGdGroup * kGdRow * 4 <= kGsSmem, "the blocks of the states have room for it");
struct GdShared {
    unsigned short list[kGcMaxDk];
    int count;
    __align__(16) float strip[kGdGroup][16];  // products of a strip's gates
};

template <bool KEYED>
__device__ __noinline__ void gd_table(const GrParams& pp, const GrChunks& ck, unsigned char* smem, GdShared& g, int block, int blocks)
{
    const GatedRecurrence& p = pp.g;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, dk = p.dk;
    // k to the end of its strip, to the end of its 32 tokens; 1 - f, q, q from its strip's start on, k
    constexpr int kArray = kGdGroup * kGdRow;
    float *near_end = reinterpret_cast<float*>(smem), *tile_end = near_end + kArray;
    const int chunks = gc_count(pp.tp.cu, pp.tp.B), pairs = chunks * ck.heads, parts = 4 * pairs <= blocks ? 4 : 2 * pairs <= blocks ? 2 : 1;
    const int c = lane, s = warp;  // a thread's channel of the group and strip while the operands are made
    bool any = false;  // most calls have none: looked for all at once (one after the other 2 x 1030 tokens of 32 heads took 137.6 us, so 133.6)
    for (int work = block + lane * blocks; work < pairs * parts; work += 32 * blocks)
        any |= ck.notes[(size_t)(work / parts / chunks) * ck.slots + work / parts % chunks].x != 0;
    if (!__any_sync(0xffffffffu, any)) return;
    for (int work = block; work < pairs * parts; work += blocks) {
        const int pair = work / parts, part = work % parts, slot = pair % chunks, h = pair / chunks;
        const size_t at = (size_t)h * ck.slots + slot;
        if (ck.notes[at].x == 0) continue;
        int b = 0, i = 0;
        (void)gc_locate(pp.tp.cu, pp.tp.B, slot, b, i);
        const int t0 = pp.tp.cu[b] + i * kGcTok, n = min(kGcTok, pp.tp.cu[b + 1] - t0);
        gs_sync();
        if (warp == 0) {
            uint32_t bits = lane < dk / 32 ? ck.fast[at * 8 + lane] : 0u;
            int to = __popc(bits);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, to, o);
                if (lane >= o) to += up;
            }
            if (lane == 31) g.count = to;
            to -= __popc(bits);
            for (; bits; bits &= bits - 1) g.list[to++] = (unsigned short)(lane * 32 + __ffs(bits) - 1);
        }
        gs_sync();
        const int channels = g.count;
        // each quarter of the SM has a strip of every 32 tokens (of some 2 or 4 parts; two or four warps to a strip then)
        const int each = 4 / parts, sub = (warp & 3) / each, I = warp >> 2, x = part + parts * ((warp & 3) % each), strip = 4 * I + x;
        const int r = lane >> 3, entry = r == x ? lane & 7 : -1;  // the lane's token lies in strip r of the strip's 32 tokens
        float acc[4][8];
#pragma unroll
        for (int e = 0; e < 4; e++)
#pragma unroll
            for (int t = 0; t < 8; t++) acc[e][t] = 0.f;
        const unsigned short *q0 = reinterpret_cast<const unsigned short*>(p.q), *k0 = reinterpret_cast<const unsigned short*>(p.k);
        unsigned short qr[8], kr[KEYED ? 8 : 1];
        float dr[8];
        auto fetch = [&](int g0) {
            const int ch = g.list[min(g0 + c, channels - 1)];
#pragma unroll
            for (int t = 0; t < 8; t++) {
                const size_t from = (size_t)(t0 + min(8 * s + t, n - 1)) * p.ld + (ck.head0 + h) * dk + ch;
                dr[t] = ck.gate[(at * kGcTok + 8 * s + t) * dk + ch];
                qr[t] = q0[from];
                if constexpr (KEYED) kr[t] = k0[from];
            }
        };
        auto value = [](unsigned short v) { return __uint_as_float((uint32_t)v << 16); };
        fetch(0);
#pragma unroll 1
        for (int g0 = 0; g0 < channels; g0 += kGdGroup) {
            gs_sync();
            const int row = c * kGdRow + 8 * s;
            auto put = [&](int array, const float(&v)[8]) {
                float* to = near_end + array * kArray + row;
                *reinterpret_cast<float4*>(to) = make_float4(v[0], v[1], v[2], v[3]);
                *reinterpret_cast<float4*>(to + 4) = make_float4(v[4], v[5], v[6], v[7]);
            };
            float end[8], left = 1.f;
            {
                float d[8], k[8], q[8], qa[8], on = 1.f;
#pragma unroll
                for (int t = 0; t < 8; t++) {
                    const bool in = g0 + c < channels && 8 * s + t < n;
                    d[t] = in ? dr[t] : 0.f;
                    k[t] = !in ? 0.f : KEYED ? value(kr[KEYED ? t : 0]) : d[t];
                    q[t] = !in ? 0.f : KEYED ? value(qr[t]) * p.q_scale : silu_of<bf16>(value(qr[t]));
                    on = fmaf(-d[t], on, on);
                    qa[t] = q[t] * on;
                }
#pragma unroll
                for (int t = 7; t >= 0; t--) {
                    end[t] = k[t] * left;
                    left = fmaf(-d[t], left, left);
                }
                g.strip[c][s] = left;
                put(0, end);
                put(2, d);
                put(3, q);
                put(4, qa);
                put(5, k);
            }
            if (g0 + kGdGroup < channels) fetch(g0 + kGdGroup);
            gs_sync();
            {
                float f = 1.f;  // from the strip's end to the end of its 32 tokens
                for (int m = s + 1; m < (s | 3) + 1; m++) f *= g.strip[c][m];
#pragma unroll
                for (int t = 0; t < 8; t++) end[t] *= f;
                put(1, end);
            }
            gs_sync();
            const int last = min(kGdGroup, channels - g0);
#pragma unroll 1
            for (int c0 = sub; c0 < last; c0 += 2 * parts) {  // two channels at a time (zeros behind the last one), for their chains' sake
                float w[2], fac[2], d[2][8], q[2][8], own_k[2];
                const float* ops[2];
                auto get = [&](float(&v)[8], const float* from) {
                    *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(from);
                    *reinterpret_cast<float4*>(v + 4) = *reinterpret_cast<const float4*>(from + 4);
                };
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    const int cc = c0 + u * parts;
                    const float4 gate = *reinterpret_cast<const float4*>(&g.strip[cc][4 * I]);
                    ops[u] = near_end + cc * kGdRow + 8 * strip;
                    w[u] = r < x ? near_end[cc * kGdRow + 32 * I + lane] : 0.f;
                    w[u] *= (r < 1 && x > 1 ? gate.y : 1.f) * (r < 2 && x > 2 ? gate.z : 1.f);
                    fac[u] = (x > 0 ? gate.x : 1.f) * (x > 1 ? gate.y : 1.f) * (x > 2 ? gate.z : 1.f);
                    own_k[u] = ops[u][5 * kArray + (lane & 7)];
                    get(d[u], ops[u] + 2 * kArray);
                    get(q[u], ops[u] + 3 * kArray);
                }
#pragma unroll
                for (int t = 0; t < 8; t++)
#pragma unroll
                    for (int u = 0; u < 2; u++) {
                        w[u] = t == entry ? own_k[u] : fmaf(-d[u][t], w[u], w[u]);
                        acc[0][t] = fmaf(q[u][t], w[u], acc[0][t]);
                    }
#pragma unroll
                for (int u = 0; u < 2; u++) get(q[u], ops[u] + 4 * kArray);
#pragma unroll
                for (int e = 1; e < 4; e++) {  // the 32 tokens e in front
                    if (e <= I) {
#pragma unroll
                        for (int u = 0; u < 2; u++) {
                            const int cc = c0 + u * parts;
                            w[u] = tile_end[cc * kGdRow + 32 * (I - e) + lane] * fac[u];
                            const float4 tile = *reinterpret_cast<const float4*>(&g.strip[cc][4 * (I - e)]);
                            fac[u] *= (tile.x * tile.y) * (tile.z * tile.w);
                        }
#pragma unroll
                        for (int t = 0; t < 8; t++) acc[e][t] = fmaf(q[1][t], w[1], fmaf(q[0][t], w[0], acc[e][t]));
                    }
                }
            }
        }
        if (parts > 1) {  // the warps of a strip
            gs_sync();
            float* sums = near_end + (I * each + (warp & 3) % each) * (parts - 1) * 1024 + lane;
            if (sub > 0) {
#pragma unroll
                for (int e = 0; e < 4; e++)
#pragma unroll
                    for (int t = 0; t < 8; t++) sums[(sub - 1) * 1024 + (e * 8 + t) * 32] = acc[e][t];
            }
            gs_sync();
            if (sub == 0) {
                for (int o = 0; o < parts - 1; o++)
#pragma unroll
                    for (int e = 0; e < 4; e++)
#pragma unroll
                        for (int t = 0; t < 8; t++) acc[e][t] += sums[o * 1024 + (e * 8 + t) * 32];
            }
        }
        if (sub == 0) {
            float* a = ck.A + (at * kGcTok + 8 * strip) * kGcTok + lane;
#pragma unroll
            for (int e = 0; e < 4; e++)
                if (e <= I) {
#pragma unroll
                    for (int t = 0; t < 8; t++) a[t * kGcTok + 32 * (I - e)] = acc[e][t];
                }
        }
    }
}

// grid: dk / COLS x dv / 128 * heads x sequences blocks for the states, the first index fastest, and the ones of gd_table behind them
template <int COLS>
__global__ void __launch_bounds__(kGsBlock, 1) gr_chunk_state_kernel(const __grid_constant__ GrParams pp, const __grid_constant__ GrChunks ck)
{
    constexpr int kCols = COLS / (kGsWarps / 4);  // channels of a thread
    const GatedRecurrence& p = pp.g;
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char *s_out = smem + kGsDepth * kGsStage, *s_vec = s_out + 3 * kGcTile;
    __shared__ __align__(8) uint64_t bars[14];  // stage is there (4), its products are done (4), accumulators are read (2), vectors are there (4)
    __shared__ uint32_t tmem_slot;
    __shared__ GdShared s_gd;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, dk = p.dk, dv = p.dv, nd = dk / 64, nv = dv / 128;
    const int states = dk / COLS * nv * ck.heads * pp.tp.B;
    if ((int)blockIdx.x >= states) {
        pdl_wait();
        pdl_launch_dependents();
        if (warp >= kGsWarps) return;
        if (p.kind == ONELLM_GR_KEYED) gd_table<true>(pp, ck, smem, s_gd, blockIdx.x - states, gridDim.x - states);
        else gd_table<false>(pp, ck, smem, s_gd, blockIdx.x - states, gridDim.x - states);
        return;
    }
    const int cols = blockIdx.x % (dk / COLS), hv = blockIdx.x / (dk / COLS) % (nv * ck.heads);
    const int slice = cols * COLS / 64, from_col = cols * COLS % 64;  // tiles have 64 channels
    const int h = ck.head0 + hv / nv, vt = hv % nv, b = blockIdx.x / (dk / COLS) / (nv * ck.heads);
    const uint32_t full0 = smem_u32(bars), done0 = smem_u32(bars + 4), free0 = smem_u32(bars + 8), vec0 = smem_u32(bars + 10);
    const uint32_t ring = smem_u32(smem);
    bool ok = (ring & 1023u) == 0;
    if (!ok && tid == 0) atomicExch(&g_tc_timeout_flag, 1);
    if (tid == 0) {
        for (int s = 0; s < 14; s++) mbar_init(full0 + 8 * s, s == 8 || s == 9 ? kGsWarps : 1);
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
    pdl_wait();
    pdl_launch_dependents();
    const int n_chunk = (pp.tp.cu[b + 1] - pp.tp.cu[b] + kGcTok - 1) / kGcTok;
    const size_t at0 = (size_t)(h - ck.head0) * ck.slots + gc_count(pp.tp.cu, b);  // behind the chunks of the sequences in front

    const int n_half = 2 * n_chunk;
    auto slot = [](int j) { return j & (kGsDepth - 1); };
    auto turn = [](int j) { return (uint32_t)(j / kGsDepth) & 1u; };
    if (warp == kGsWarps) {
        const bool leader = elect_one();
        int loaded = 0;
        // half a chunk; with the first one the chunk's vectors, whose place is free: the products waited for were issued behind the wait for
        // the warps that read them
        for (int j = 0; j < n_half && ok; j++) {
            if (j >= kGsDepth) ok = mbar_wait_warp(done0 + 8 * slot(j), turn(j - kGsDepth));
            if (!ok) break;
            if (leader) {
                const size_t at = at0 + (j >> 1);
                const int from = (j & 1) * kGsHalf;
                if (!(j & 1)) {
                    const int i = (j >> 1) & 3;
                    mbar_expect_tx(vec0 + 8 * i, kGsVec);
                    bulk_load(smem_u32(s_vec) + i * kGsVec, ck.vec + (at * nd + slice) * 256, kGsVec, vec0 + 8 * i);
                }
                const uint32_t dst = ring + slot(j) * kGsStage, bar = full0 + 8 * slot(j);
                mbar_expect_tx(bar, kGsStage);
                for (int e = 0; e < 2; e++) bulk_load(dst + e * kGsHalf, ck.v + ((at * nv + vt) * 2 + e) * kGcTile + from, kGsHalf, bar);
                for (int e = 0; e < 3; e++) bulk_load(dst + (2 + e) * kGsHalf, ck.k + ((at * nd + slice) * 3 + e) * kGcTile + from, kGsHalf, bar);
            }
            loaded = j + 1;
            __syncwarp();
        }
        if (!ok) {  // what is on its way ends before the block does
            ring_drain(full0, kGsDepth, loaded);
            ring_drain(vec0, 4, (loaded + 1) / 2);
        }
    } else if (warp == kGsWarps + 1) {
        const bool leader = elect_one();
        // D[value, channel] += V^T k~: the tokens are the rows of both operands as they lie in memory
        const uint32_t idesc = (1u << 4) | umma_operand_bits<bf16>() | (1u << 15) | (1u << 16) | ((COLS >> 3) << 17) | ((128u >> 4) << 24);
        const uint64_t da = umma_desc(ring, kGsHalf, 1024), db = umma_desc(ring + 2 * kGsHalf + from_col * 2, kGsHalf, 1024);
        int issued = 0;
        for (int j = 0; j < n_half && ok; j++) {
            const int i = j >> 1;
            if (!(j & 1) && i >= 2) ok = mbar_wait_warp(free0 + 8 * (i & 1), (uint32_t)((i >> 1) - 1) & 1u);
            ok = ok && mbar_wait_warp(full0 + 8 * slot(j), turn(j));
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (leader) {
                const uint64_t st = (uint64_t)((slot(j) * kGsStage) >> 4);
#pragma unroll
                for (int q = 0; q < 2; q++)  // an accumulator for every 32 tokens
#pragma unroll
                    for (int e = 2; e >= 0; e--)
#pragma unroll
                        for (int kk = 0; kk < 2; kk++)
                            umma_f16(tmem + (uint32_t)((i & 1) * 4 * COLS + ((j & 1) * 2 + q) * COLS), da + st + (uint64_t)((q * 4096 + kk * 2048) >> 4),
                                     db + st + (uint64_t)((e * kGsHalf + q * 4096 + kk * 2048) >> 4), idesc, e < 2 || kk > 0 ? 1u : 0u);
                umma_commit(done0 + 8 * slot(j));
            }
            issued = j + 1;
            __syncwarp();
        }
        if (!ok) ring_drain(done0, kGsDepth, issued);
    } else if (ok && n_chunk > 0) {
        const int q = warp & 3, part = warp >> 2, row = q * 32 + lane, v = vt * 128 + row, c0 = part * kCols;
        const uint32_t t_lane = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)c0;
        float* state = p.state + (((size_t)b * p.H + h) * dk + cols * COLS + c0) * dv + v;
        const bool fresh = pp.tp.hist[b] == 0;
        float S[kCols];
        auto is_rare = [&](size_t at) { return (ck.notes[at].y | ck.notes[at].z | ck.notes[at].w) != 0; };
        bool rare = is_rare(at0);
#pragma unroll
        for (int c = 0; c < kCols; c++) S[c] = fresh ? 0.f : state[(size_t)c * dv];
        for (int i = 0; i < n_chunk; i++) {
            const size_t at = at0 + i;
            const bool next = i + 1 < n_chunk && is_rare(at + 1);
            bool there = ok && mbar_wait_warp(vec0 + 8 * (i & 3), (uint32_t)(i >> 2) & 1u);
            const float4* vec = reinterpret_cast<const float4*>(s_vec + (i & 3) * kGsVec) + (from_col + c0) / 4;  // + 16: the next vector
            // the pieces of the chunk in front have been read out of shared memory before anyone writes the next ones; half rows have two places
            const int place = COLS == 64 ? 0 : (i & 1) * 32;
            if constexpr (COLS == 64) {
                if (tid == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                gs_sync();
            }
#pragma unroll
            for (int g = 0; g < kCols / 8; g++) {
                uint32_t p0[4], p1[4], p2[4], rest = 0u;
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const float4 bm = vec[2 * g + e];
                    const float* x = S + 8 * g + 4 * e;
                    split_pair(x[0] * bm.x, x[1] * bm.y, p0[2 * e], p1[2 * e], p2[2 * e], rest);
                    split_pair(x[2] * bm.z, x[3] * bm.w, p0[2 * e + 1], p1[2 * e + 1], p2[2 * e + 1], rest);
                }
                unsigned char* dst = s_out + gc_at(row, place + c0 + 8 * g);
                *reinterpret_cast<uint4*>(dst) = make_uint4(p0[0], p0[1], p0[2], p0[3]);
                *reinterpret_cast<uint4*>(dst + kGcTile) = make_uint4(p1[0], p1[1], p1[2], p1[3]);
                *reinterpret_cast<uint4*>(dst + 2 * kGcTile) = make_uint4(p2[0], p2[1], p2[2], p2[3]);
            }
            unsigned char* out = ck.s + ((at * nv + vt) * nd + slice) * 3 * kGcTile;
            if constexpr (COLS == 64) {
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                gs_sync();
                if (tid == 0) {
                    bulk_store(out, smem_u32(s_out), 3 * kGcTile);
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
            } else {
                gs_sync();
#pragma unroll
                for (int e = 0; e < 3; e++)  // four threads to the 64 bytes of a row
                    *reinterpret_cast<uint4*>(out + e * kGcTile + gc_at(tid >> 2, from_col + (tid & 3) * 8)) =
                        *reinterpret_cast<const uint4*>(s_out + e * kGcTile + gc_at(tid >> 2, place + (tid & 3) * 8));
            }
            there = there && mbar_wait_warp(done0 + 8 * slot(2 * i + 1), turn(2 * i + 1));
            if (!there) ok = false;  // goes on to the barriers of the others, with nothing stored at the end
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t acc = t_lane + (uint32_t)((i & 1) * 4 * COLS);
            auto sums = [&](int e, float(&two)[kCols]) {  // of 64 tokens
                uint32_t x[kCols], y[kCols];
                if constexpr (kCols == 16) {
                    tmem_ld16(acc + (uint32_t)(e * COLS), x);
                    tmem_ld16(acc + (uint32_t)(e * COLS + COLS), y);
                } else {
                    tmem_ld8(acc + (uint32_t)(e * COLS), x);
                    tmem_ld8(acc + (uint32_t)(e * COLS + COLS), y);
                }
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int c = 0; c < kCols; c++) two[c] = __uint_as_float(x[c]) + __uint_as_float(y[c]);
            };
            float add[kCols], more[kCols];
            sums(0, add);
            sums(2, more);
            if (!rare) {
#pragma unroll
                for (int e = 0; e < kCols / 4; e++) {
                    const float4 be = vec[16 + e], al = vec[32 + e], ga = vec[48 + e];
                    const float fe[4] = {be.x, be.y, be.z, be.w}, fa[4] = {al.x, al.y, al.z, al.w}, fg[4] = {ga.x, ga.y, ga.z, ga.w};
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const int c = 4 * e + j;
                        S[c] = fmaf(fe[j], add[c] + more[c], fmaf(fa[j], S[c], fg[j] * S[c]));
                    }
                }
            } else {  // values that are not finite, or have been divided: each half's sums by themselves, behind their factor
                const float* f = reinterpret_cast<const float*>(vec);
                const int4 notes = ck.notes[at];
                const bool bad = (notes.y && ck.bad[at * 2 * dv + v] < kGcTok) || (notes.z && ck.bad[(at * 2 + 1) * dv + v] < kGcTok);
#pragma unroll
                for (int c = 0; c < kCols; c++) {
                    const float kept = fmaf(f[128 + c], S[c], f[192 + c] * S[c]);
                    S[c] = bad       ? __uint_as_float(0x7fffffffu)
                           : notes.w ? fmaf(f[64 + c] * add[c], two_to(notes.w & 0xffff), fmaf(f[64 + c] * more[c], two_to(notes.w >> 16), kept))
                                     : fmaf(f[64 + c], add[c] + more[c], kept);
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(free0 + 8 * (i & 1));  // the accumulators and the vectors
            rare = next;
        }
        if (ok) {
#pragma unroll
            for (int c = 0; c < kCols; c++) state[(size_t)c * dv] = S[c];
        }
        if (COLS == 64 && tid == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

// ---- 3. the outputs ------------------------------------------------------------------------------------------
constexpr int kGoWarps = 8;
constexpr int kGoBlock = kGoWarps * 32 + 64;  // and one that issues the loads, one the products
constexpr int kGoRing = 14;                   // tiles on their way or in use
constexpr int kGoSmem = kGoRing * kGcTile;
// Tensor memory: q~ . k~ (large and small products), q~ . S (the same).  The pieces of 16 tokens of the table lie over the columns that
// these came from; its product with V adds to the small ones.
constexpr uint32_t kGoTable = 0, kGoTableLow = 128, kGoState = 256, kGoStateLow = 384;

__device__ __forceinline__ void go_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kGoWarps * 32) : "memory"); }  // the warps that make the output
// grid (dv / 128, clusters), cluster (dv / 128, 1, 1): a cluster has the value tiles of a head and takes every gridDim.y-th pair of chunk and head
__global__ void __launch_bounds__(kGoBlock, 1) gr_chunk_output_kernel(const __grid_constant__ GrParams pp, const __grid_constant__ GrChunks ck)
{
    const GatedRecurrence& p = pp.g;
    extern __shared__ __align__(1024) unsigned char smem[];
    // tile is there (14), tile has been used (14), table is done, pieces of the table are there, output is done, output is read, sums of the
    // cluster are there, everything issued by a block that gave up is done, products with the state are done
    __shared__ __align__(8) uint64_t bars[2 * kGoRing + 7];
    __shared__ uint32_t tmem_slot;
    __shared__ float s_part[kGcTok], s_sum[2][kGcTok], s_w[128];
    cg::cluster_group cluster = cg::this_cluster();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, dk = p.dk, dv = p.dv, nd = dk / 64, nv = dv / 128;
    const int vt = blockIdx.x;
    const uint32_t full0 = smem_u32(bars), used0 = full0 + 8 * kGoRing, t_done = used0 + 8 * kGoRing, p_full = t_done + 8, o_done = t_done + 16,
                   o_read = t_done + 24, sums = t_done + 32, end = t_done + 40, s_done = t_done + 48;
    const uint32_t ring = smem_u32(smem);
    bool ok = (ring & 1023u) == 0;
    if (!ok && tid == 0) atomicExch(&g_tc_timeout_flag, 1);
    if (tid == 0) {
        for (int s = 0; s < 2 * kGoRing + 7; s++) {
            const int e = s - 2 * kGoRing;
            mbar_init(full0 + 8 * s, e == 1 || e == 3 ? kGoWarps : e == 4 ? kGoWarps * nv : 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    cluster.sync();  // the peers' barriers too
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    // No block of this kernel starts before every block of the state kernel is behind its wait for the prepare kernel: what that one wrote
    // is there.  The wait for the states comes in front of their first load (and of the first store).
    const int chunks = gc_count(pp.tp.cu, pp.tp.B);
    const long n_work = (long)chunks * ck.heads;
    const int mine = n_work > blockIdx.y ? (int)((n_work - 1 - blockIdx.y) / gridDim.y) + 1 : 0;  // the same in all blocks of a cluster
    auto place = [&](int k, int& s, int& h) {  // of the k-th pair of this cluster
        const long w = blockIdx.y + (long)k * gridDim.y;
        s = (int)(w % chunks);
        h = ck.head0 + (int)(w / chunks);
        return (size_t)(h - ck.head0) * ck.slots + s;
    };

    // The tiles of a pair in the order of their use: of 64 channels q~0 k~0 k~1 q~1 k~2 q~2 S0 S1 S2 (pieces), then of the next; V at the end.
    if (warp == kGoWarps) {
        const bool leader = elect_one();
        int slot = 0, loaded = 0;
        uint32_t phase = 1;  // of the places' last use
        auto load = [&](const unsigned char* src) {
            if (!ok) return;
            if (loaded >= kGoRing) ok = mbar_wait_warp(used0 + 8 * slot, phase);
            if (!ok) return;
            if (leader) {
                mbar_expect_tx(full0 + 8 * slot, kGcTile);
                bulk_load(ring + slot * kGcTile, src, kGcTile, full0 + 8 * slot);
            }
            __syncwarp();
            loaded++;
            if (++slot == kGoRing) {
                slot = 0;
                phase ^= 1;
            }
        };
        for (int k = 0; k < mine && ok; k++) {
            int s, h;
            const size_t at = place(k, s, h);
#pragma unroll 1
            for (int d = 0; d < nd && ok; d++) {
                const unsigned char *q = ck.q + (at * nd + d) * 3 * kGcTile, *kt = ck.k + (at * nd + d) * 3 * kGcTile,
                                    *st = ck.s + ((at * nv + vt) * nd + d) * 3 * kGcTile;
                load(q);
                load(kt);
                load(kt + kGcTile);
                load(q + kGcTile);
                load(kt + 2 * kGcTile);
                load(q + 2 * kGcTile);
                if (k == 0 && d == 0) pdl_wait();
#pragma unroll 1
                for (int e = 0; e < 3; e++) load(st + e * kGcTile);
            }
#pragma unroll 1
            for (int e = 0; e < 2; e++) load(ck.v + ((at * nv + vt) * 2 + e) * kGcTile);
        }
        if (!ok) {  // what is on its way ends before the block does
            ring_drain(full0, kGoRing, loaded);
        }
    } else if (warp == kGoWarps + 1) {
        const bool leader = elect_one();
        const uint32_t types = (1u << 4) | umma_operand_bits<bf16>() | ((128u >> 4) << 24), square = types | ((128u >> 3) << 17);
        const uint64_t d0 = umma_desc(ring, 16, 1024), dv0 = umma_desc(ring, kGcTile, 1024);
        int slot = 0;  // of the next tile
        uint32_t phase = 0;
        bool issued = false;
        // waits for the next tile and says where it is
        auto next = [&]() {
            const int at = slot;
            ok = ok && mbar_wait_warp(full0 + 8 * slot, phase);
            if (++slot == kGoRing) {
                slot = 0;
                phase ^= 1;
            }
            return at;
        };
        auto product = [&](int a, int b, uint32_t to, uint32_t accumulate) {  // 64 channels
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (ok && leader) {
                const uint64_t da = d0 + (uint64_t)(a * (kGcTile >> 4)), db = d0 + (uint64_t)(b * (kGcTile >> 4));
#pragma unroll
                for (int kk = 0; kk < 4; kk++) umma_f16(tmem + to, da + (uint64_t)((kk * 32) >> 4), db + (uint64_t)((kk * 32) >> 4), square, kk > 0 ? 1u : accumulate);
            }
            issued = true;
            __syncwarp();
        };
        auto release = [&](int a) {
            if (ok && leader) umma_commit(used0 + 8 * a);
            __syncwarp();
        };
        // Only MMAs of the same shape and accumulator are promised to run in the order of their issue.  Two places need another order and wait: the
        // table's product of a pair overwrites the pieces that the last one of the pair in front reads, and that one, 64 columns wide, adds to sums of
        // products 128 wide.
        for (int k = 0; k < mine && ok; k++) {
            if (k > 0) ok = mbar_wait_warp(o_done, (uint32_t)(k - 1) & 1u);
#pragma unroll 1
            for (int d = 0; d < nd && ok; d++) {
                const uint32_t more = d > 0;
                const int q0 = next(), k0 = next();
                product(q0, k0, kGoTable, more);
                const int k1 = next();
                product(q0, k1, kGoTableLow, more);
                const int q1 = next();
                product(q1, k0, kGoTableLow, 1u);
                product(q1, k1, kGoTableLow, 1u);
                release(k1);
                const int k2 = next();
                product(q0, k2, kGoTableLow, 1u);
                release(k2);
                const int q2 = next();
                product(q2, k0, kGoTableLow, 1u);
                release(k0);
                if (d == nd - 1) {
                    if (ok && leader) umma_commit(t_done);
                    __syncwarp();
                }
                if (d == 0 && k > 0) ok = ok && mbar_wait_warp(o_read, (uint32_t)(k - 1) & 1u);
                const int s0 = next();
                product(q0, s0, kGoState, more);
                product(q2, s0, kGoStateLow, more);
                release(q2);
                product(q1, s0, kGoStateLow, 1u);
                const int s1 = next();
                product(q0, s1, kGoStateLow, 1u);
                product(q1, s1, kGoStateLow, 1u);
                release(q1);
                release(s1);
                release(s0);
                const int s2 = next();
                product(q0, s2, kGoStateLow, 1u);
                if (d == nd - 1) {
                    if (ok && leader) umma_commit(s_done);
                    __syncwarp();
                }
                release(q0);
                release(s2);
            }
            const int v0 = next(), v1 = next();
            ok = ok && mbar_wait_warp(s_done, (uint32_t)k & 1u) && mbar_wait_warp(p_full, (uint32_t)k & 1u);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (leader) {
                const uint32_t idesc = types | (1u << 16) | ((64u >> 3) << 17);
#pragma unroll 1
                for (int e = 5; e >= 0; e--) {  // the third pieces with both halves of the columns first
                    const uint32_t table = e >= 4 ? kGoTableLow : kGoTable + 8u * (uint32_t)(e >> 1);
                    const uint64_t dv = dv0 + (uint64_t)((e & 1 ? v1 : v0) * (kGcTile >> 4));
#pragma unroll
                    for (int kk = 0; kk < 8; kk++)
                        umma_f16_tmem_a(tmem + kGoStateLow + 64u * (uint32_t)(e & 1), tmem + table + (uint32_t)(kk * 16), dv + (uint64_t)((kk * 2048) >> 4), idesc,
                                        1u);
                }
                umma_commit(used0 + 8 * v0);
                umma_commit(used0 + 8 * v1);
                umma_commit(o_done);
            }
            __syncwarp();
        }
        if (!ok && issued) {
            if (leader) umma_commit(end);
            __syncwarp();
            (void)mbar_wait(end, 0);
        }
    } else {
        const int q = warp & 3, half = warp >> 2, row = q * 32 + lane;  // a thread has a token and 64 of the columns
        const uint32_t t_lane = tmem + ((uint32_t)(q * 32) << 16);
        pdl_launch_dependents();
        if (mine == 0) pdl_wait();
        if (tid < 128) s_w[tid] = p.w[vt * 128 + tid];
        go_sync();
        for (int k = 0; k < mine; k++) {
            int s, h, b = 0, i = 0;
            const size_t at = place(k, s, h);
            const uint32_t phase = (uint32_t)k & 1u;
            (void)gc_locate(pp.tp.cu, pp.tp.B, s, b, i);
            const int t0 = pp.tp.cu[b] + i * kGcTok, n = min(kGcTok, pp.tp.cu[b + 1] - t0);
            const int4 notes = ck.notes[at];
            if (k == 0 && notes.x) pdl_wait();  // the state kernel has made a table
            if (ok) ok = mbar_wait_warp(t_done, phase);
            if (ok) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const int last = row < n ? row : -1;  // the tokens this one sees
#pragma unroll 1
                for (int j0 = half * 64; j0 < half * 64 + 64; j0 += 16) {
                    uint32_t x[16], y[16], p0[8], p1[8], p2[8], rest = 0u;
                    tmem_ld16(t_lane + kGoTable + (uint32_t)j0, x);
                    tmem_ld16(t_lane + kGoTableLow + (uint32_t)j0, y);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    float a[16];
#pragma unroll
                    for (int j = 0; j < 16; j++) a[j] = __uint_as_float(x[j]) + __uint_as_float(y[j]);
                    if (notes.x) {
                        const float* src = ck.A + (at * kGcTok + row) * kGcTok + j0;
#pragma unroll
                        for (int j = 0; j < 16; j++)
                            if (j0 + j <= last) a[j] = notes.x == 1 ? src[j] : a[j] + src[j];
                    }
                    if (notes.w) {  // a warp's columns are the tokens of one of the halves
#pragma unroll
                        for (int j = 0; j < 16; j++) a[j] *= two_to(half ? notes.w >> 16 : notes.w & 0xffff);
                    }
#pragma unroll
                    for (int j = 0; j < 8; j++)
                        split_pair(j0 + 2 * j <= last ? a[2 * j] : 0.f, j0 + 2 * j + 1 <= last ? a[2 * j + 1] : 0.f, p0[j], p1[j], p2[j], rest);
                    tmem_st8(t_lane + kGoTable + (uint32_t)j0, p0);
                    tmem_st8(t_lane + kGoTable + (uint32_t)j0 + 8u, p1);
                    tmem_st8(t_lane + kGoTableLow + (uint32_t)j0, p2);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(p_full);
            }
            if (k == 0) pdl_wait();
            const size_t col = (size_t)h * dv + vt * 128 + half * 64;
            if (ok) ok = mbar_wait_warp(o_done, phase);
            float o[64], ss = -1.f;
            if (ok) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                ss = 0.f;
#pragma unroll
                for (int g = 0; g < 4; g++) {
                    uint32_t x[16], y[16];
                    tmem_ld16(t_lane + kGoState + (uint32_t)(half * 64 + g * 16), x);
                    tmem_ld16(t_lane + kGoStateLow + (uint32_t)(half * 64 + g * 16), y);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int j = 0; j < 16; j++) o[g * 16 + j] = __uint_as_float(x[j]) + __uint_as_float(y[j]);
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(o_read);
                for (int e = 0; e < 2; e++) {
                    if (!(e ? notes.z : notes.y)) continue;
                    const int* bad = ck.bad + (at * 2 + e) * dv + vt * 128 + half * 64;
#pragma unroll
                    for (int j = 0; j < 64; j++)
                        if (bad[j] <= row) o[j] = __uint_as_float(0x7fffffffu);
                }
#pragma unroll
                for (int j = 0; j < 64; j++) ss = fmaf(o[j], o[j], ss);
            }
            // The sums of a pair lie with each block and are read by all; they are written over two pairs later, when every warp of the cluster
            // has come to the pair between.  Below zero: that block gave up, and nothing of the cluster's pair is stored.
            if (half == 1) s_part[row] = ss;
            go_sync();
            if (half == 0) s_sum[phase][row] = ss < 0.f || s_part[row] < 0.f ? -1.f : ss + s_part[row];
            float all = 0.f;
            bool store = true;
            if (nv > 1) {
                __syncwarp();
                if (lane < nv) mbar_arrive_cluster(map_to_rank(sums, (uint32_t)lane));
                store = __all_sync(0xffffffffu, mbar_wait_cluster(sums, phase));
                ok = ok && store;
            } else {
                go_sync();
            }
            for (int r = 0; r < nv; r++) {
                const float part = *cluster.map_shared_rank(&s_sum[phase][row], r);
                store &= !(part < 0.f);
                all += part;
            }
            if (store && row < n) {
                const float inv = p.out_scale / sqrtf(all / (float)p.norm_width + p.eps);
                bf16* dst = reinterpret_cast<bf16*>(p.out) + (size_t)(t0 + row) * p.out_ld + col;
                const bf16* gp = p.g ? reinterpret_cast<const bf16*>(p.g) + (size_t)(t0 + row) * p.ld + col : nullptr;
#pragma unroll
                for (int c = 0; c < 64; c += 16) {
                    if (gp) {
                        float f[2][8];
                        Vec16<bf16>::load(gp + c, f[0]);
                        Vec16<bf16>::load(gp + c + 8, f[1]);
#pragma unroll
                        for (int j = 0; j < 16; j++) o[c + j] = o[c + j] * inv * s_w[half * 64 + c + j] * silu_of<bf16>(f[j >> 3][j & 7]);
                    } else {
#pragma unroll
                        for (int j = 0; j < 16; j++) o[c + j] = o[c + j] * inv * s_w[half * 64 + c + j];
                    }
                    *reinterpret_cast<uint4*>(dst + c) = Vec16<bf16>::pack(*reinterpret_cast<float(*)[8]>(o + c));
                    *reinterpret_cast<uint4*>(dst + c + 8) = Vec16<bf16>::pack(*reinterpret_cast<float(*)[8]>(o + c + 8));
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    cluster.sync();  // peers may still be writing sums into this block's memory
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}
static const TimeoutFlag timeout_flag(tc_flag_read_clear, tc_flag_address);

// ---- host ----------------------------------------------------------------------------------------------------
// Tokens of a sequence on average from which the chunks are the faster form.  The three launches take 30 to 55 us however few chunks there are;
// token by token a call takes 0.11 to 0.22 us a token, and twice that where its blocks (32 columns of a head each) are more than the SMs.
// us, token by token | in chunks: TIED 128 x 128, 16 heads, 1 x 256 tokens 37.9 | 32.0, 8 x 192 tokens 96.6 | 69.6, 2 x 160 (128 blocks) 30.1 |
// 34.3; KEYED 256 x 512, 8 heads, 1 x 256 76 | 57, 8 x 192 330 | 212; KEYED 64 x 128, 2 heads, 8 x 256 (64 blocks) 36.2 | 37.3.
constexpr int kGcLeastTokens = 288, kGcLeastTokensFull = 192;

static long gc_slots(int tokens, int B) { return (long)tokens / kGcTok + B; }

// Heads that go through the three launches together, 0: the call is not for them.  A chunk of a head takes 1.7 to 2.1 times the token by token form's
// vectors of it, and more where sequences end within chunks, so a call takes no more than the larger of that form's work space and kGcSpace, and
// goes through its heads in passes where all of them would need more.  With 256 MB, 8 x 512 tokens of 32 heads of 128 x 128 went in three passes, 302 us
// instead of 233.
constexpr size_t kGcSpace = (size_t)1 << 30;
constexpr size_t kGcPad = 10 * 16;  // the parts of the work space begin on multiples of 16 bytes
static int gc_heads(int kind, int tokens, int B, int H, int dk, int dv)
{
    const size_t space = gated_recurrence_workspace(kind, tokens, H, dk, dv) - kGcPad, head = (size_t)gc_slots(tokens, B) * gc_chunk_bytes(dk, dv);
    const int most = (int)std::min<size_t>(space / head, H), passes = most > 0 ? (H + most - 1) / most : 0;
    return passes > 0 ? (H + passes - 1) / passes : 0;
}

size_t gr_chunked_workspace(int tokens, int H, int dk, int dv)
{
    if (dk % 64 != 0 || dk > kGcMaxDk || dv % 128 != 0 || dv > kGcMaxDv || tokens < kGcLeastTokensFull) return 0;
    return std::min(kGcSpace, (size_t)gc_slots(tokens, tokens / kGcLeastTokensFull) * H * gc_chunk_bytes(dk, dv) + kGcPad);
}

bool gr_chunked_takes(const GatedRecurrence& g, const TokenPositions& tp, int B, int tokens)
{
    const auto multiple = [](const void* p, uintptr_t n) { return reinterpret_cast<uintptr_t>(p) % n == 0; };
    const bool keyed = g.kind == ONELLM_GR_KEYED;
    const int least = (long)B * g.H * (g.dv / 32) > num_sms() ? kGcLeastTokensFull : kGcLeastTokens;
    return g.dtype == ONELLM_BF16 && tp.cu && g.dk % 64 == 0 && g.dk <= kGcMaxDk && g.dv % 128 == 0 && g.dv <= kGcMaxDv && (!keyed || g.rank <= kGcMaxRank) &&
           (long)tokens >= (long)least * B && gc_slots(tokens, B) < (1 << 24) && g.H <= 65535 && (long)g.H * (g.dv / 128) * (g.dk / 32) * B < (1 << 30) && multiple(g.q, 4) &&
           multiple(keyed ? g.k : g.z, 4) && multiple(g.v, 8) && multiple(g.zb, 8) && multiple(keyed ? g.A : g.lower, 16) && multiple(g.g, 16) &&
           multiple(g.out, 16) && g.out_ld % 8 == 0 && gc_heads(g.kind, tokens, B, g.H, g.dk, g.dv) > 0;
}

// Clusters of `nv` output blocks that run at once, asked once per device: a GPC of 18 SMs has room for four clusters of four, and a
// cluster more than there is room for would run when the others are through (4 heads of 256 x 512, 2 x 1030 tokens, 37 clusters where 34 run at
// once: all three launches 144 us instead of 119).
static int go_clusters(int nv)
{
    static std::mutex mu;
    static int known[kMaxDevices][kGcMaxDv / 128 + 1] = {};
    std::lock_guard<std::mutex> lock(mu);
    int& n = known[current_device()][nv];
    if (n == 0) {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute a[1];
        a[0].id = cudaLaunchAttributeClusterDimension;
        a[0].val.clusterDim.x = nv;
        a[0].val.clusterDim.y = 1;
        a[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3(nv, 1024);
        cfg.blockDim = dim3(kGoBlock);
        cfg.dynamicSmemBytes = kGoSmem;
        cfg.attrs = a;
        cfg.numAttrs = 1;
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, gr_chunk_output_kernel, &cfg) != cudaSuccess || clusters < 1) {
            (void)cudaGetLastError();
            clusters = num_sms() / nv;
        }
        n = std::max(1, clusters);
    }
    return n;
}

template <typename... KArgs, typename... Args>
static cudaError_t gc_launch(void (*kern)(KArgs...), dim3 grid, int threads, size_t smem, dim3 cluster, cudaStream_t st, Args... args)
{
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute a[2];
    a[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a[0].val.programmaticStreamSerializationAllowed = 1;
    a[1].id = cudaLaunchAttributeClusterDimension;
    a[1].val.clusterDim.x = cluster.x;
    a[1].val.clusterDim.y = cluster.y;
    a[1].val.clusterDim.z = cluster.z;
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = a;
    cfg.numAttrs = 2;
    note_launch();
    return cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}

int gr_chunked(const GrParams& p, int B, int tokens, cudaStream_t st)
{
    const GatedRecurrence& g = p.g;
    const bool keyed = g.kind == ONELLM_GR_KEYED;
    const int dk = g.dk, dv = g.dv, slots = (int)gc_slots(tokens, B), nv = dv / 128, heads = gc_heads(g.kind, tokens, B, g.H, dk, dv);
    const size_t n = (size_t)slots * heads;
    GrChunks ck;
    ck.slots = slots;
    unsigned char* w = static_cast<unsigned char*>(g.work);
    auto take = [&](size_t bytes) {
        unsigned char* r = w;
        w += (n * bytes + 15) / 16 * 16;
        return r;
    };
    ck.q = take((size_t)3 * kGcTok * dk * 2);
    ck.k = take((size_t)3 * kGcTok * dk * 2);
    ck.s = take((size_t)3 * dv * dk * 2);
    ck.v = take((size_t)kGcTok * dv * 2);
    ck.vec = reinterpret_cast<float*>(take((size_t)4 * dk * 4));
    ck.A = reinterpret_cast<float*>(take((size_t)kGcTok * kGcTok * 4));
    ck.bad = reinterpret_cast<int*>(take((size_t)2 * dv * 4));
    ck.gate = reinterpret_cast<float*>(take((size_t)4 * kGcTok * dk));
    ck.fast = reinterpret_cast<uint32_t*>(take(32));
    ck.notes = reinterpret_cast<int4*>(take(16));

    const size_t prep = (size_t)kGcTok / 2 * (dk + (keyed ? g.rank : 0)) * sizeof(float);
    auto k1 = keyed ? gr_chunk_prepare_kernel<true> : gr_chunk_prepare_kernel<false>;
    static DeviceOnce attr;
    ONELLM_CUDA(attr.run([] {
        cudaError_t e = cudaFuncSetAttribute(gr_chunk_prepare_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGcTok / 2 * (kGcMaxDk + kGcMaxRank) * 4);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(gr_chunk_prepare_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGcTok / 2 * (kGcMaxDk + kGcMaxRank) * 4);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(gr_chunk_state_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGsSmem);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(gr_chunk_state_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGsSmem);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(gr_chunk_output_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kGoSmem);
        for (const void* k : {(const void*)gr_chunk_prepare_kernel<true>, (const void*)gr_chunk_prepare_kernel<false>, (const void*)gr_chunk_state_kernel<64>,
                              (const void*)gr_chunk_state_kernel<32>,
                              (const void*)gr_chunk_output_kernel})
            if (e == cudaSuccess) e = prefer_max_shared(k);
        return e;
    }));
    for (ck.head0 = 0; ck.head0 < g.H; ck.head0 += heads) {
        ck.heads = std::min(heads, g.H - ck.head0);
        const long clusters = std::min((long)go_clusters(nv), (long)slots * ck.heads);
        // 32 channels a block where there is an SM for each of them: a chunk's step is as long as the work of a thread
        const bool narrow = (long)(dk / 32) * nv * ck.heads * B <= num_sms();
        const unsigned states = (unsigned)(dk / (narrow ? 32 : 64) * nv * ck.heads * B);
        ONELLM_CUDA(gc_launch(k1, dim3(slots, ck.heads, 4), 2 * dk, prep, dim3(1, 1, 2), st, p, ck));
        ONELLM_CUDA(gc_launch(narrow ? gr_chunk_state_kernel<32> : gr_chunk_state_kernel<64>, dim3(states + num_sms()), kGsBlock, kGsSmem, dim3(1), st, p, ck));
        ONELLM_CUDA(gc_launch(gr_chunk_output_kernel, dim3(nv, (unsigned)clusters), kGoBlock, kGoSmem, dim3(nv), st, p, ck));
    }
    return ONELLM_OK;
}

}  // namespace onellm
