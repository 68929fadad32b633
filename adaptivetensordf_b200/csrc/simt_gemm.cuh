// Register-tiled FP32 products of small matrices in shared memory, for the
// decoder MLP on the CUDA cores (fused_simt.cuh, mlp.cu).
//
// Every operand is stored with the contraction index contiguous, so a thread
// loads four of its values per row with one 16-byte load and multiplies them
// as two packed pairs (fma.rn.f32x2): a pair accumulates the even and the odd
// terms, added at the end. Each lane is a plain FP32 fma.
//
// Lanes of a warp: bits 0, 3, 4 of the lane pick the rows (A), bits 1, 2 the
// columns (B): lane_row, lane_col. On sm_100a a warp's 16-byte shared load
// takes 2.1 cycles when either neighbouring lanes or every other lane of each
// 8 read the same address, and 3.9 otherwise; with this mapping both operands'
// loads are of the cheap kind (lane / 4 and lane % 4 left B's at 3.9). An
// 8 x 4 tile of outputs per thread costs 12 * 2.1 = 25 load cycles per 4 steps
// of the contraction against 32 cycles of its 128 FMAs per lane at 128 a
// cycle; a smaller tile would be bound by the loads. Rows and columns of a
// thread are interleaved (row i * groups + group), and the pitches are 4 mod
// 32 floats (or 12, 20, 28) apart, so the distinct addresses of a load fall
// into distinct banks.
#pragma once

#include <stdint.h>

#include "atdf_common.cuh"

namespace atdf {

__device__ __forceinline__ int lane_row(int lane) { return (lane & 1) | ((lane >> 3) << 1); }  // 0..7
__device__ __forceinline__ int lane_col(int lane) { return (lane >> 1) & 3; }                     // 0..3

// Sum over the 4 lanes that share a row.
__device__ __forceinline__ float sum_cols(float v)
{
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    return v + __shfl_xor_sync(0xffffffffu, v, 4);
}

// Sum over the 8 lanes that share a column.
__device__ __forceinline__ float sum_rows(float v)
{
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    v += __shfl_xor_sync(0xffffffffu, v, 8);
    return v + __shfl_xor_sync(0xffffffffu, v, 16);
}

__device__ __forceinline__ uint64_t ffma2(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

__device__ __forceinline__ uint64_t pack2(float lo, float hi)
{
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}

__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}

__device__ __forceinline__ float sum2(uint64_t v)
{
    float lo, hi;
    unpack2(v, lo, hi);
    return lo + hi;
}

// acc[i][j] += sum_k a[i * a_step + k] * b[j * b_step + k] over K (a multiple
// of 4) contiguous k; a and b point at the thread's first row and column.
template <int RM, int CN, int K>
__device__ __forceinline__ void gemm_k(uint64_t (&acc)[RM][CN], const float* a, int a_step, const float* b,
                                       int b_step)
{
#pragma unroll 2
    for (int k = 0; k < K; k += 4) {
        ulonglong2 av[RM], bv[CN];
#pragma unroll
        for (int i = 0; i < RM; ++i) av[i] = *reinterpret_cast<const ulonglong2*>(a + i * a_step + k);
#pragma unroll
        for (int j = 0; j < CN; ++j) bv[j] = *reinterpret_cast<const ulonglong2*>(b + j * b_step + k);
#pragma unroll
        for (int i = 0; i < RM; ++i)
#pragma unroll
            for (int j = 0; j < CN; ++j) {
                acc[i][j] = ffma2(av[i].x, bv[j].x, acc[i][j]);
                acc[i][j] = ffma2(av[i].y, bv[j].y, acc[i][j]);
            }
    }
}

// acc[i][j] += sum_s (a[s][2 i], a[s][2 i + 1]) * b[s][j]: a weight gradient
// over S samples, both operands sample-major with 2 RP and CN contiguous
// values per thread; the pairs run along a's columns.
template <int RP, int CN>
__device__ __forceinline__ void gemm_s(uint64_t (&acc)[RP][CN], const float* a, int a_pitch, const float* b,
                                       int b_pitch, int S)
{
    static_assert(RP % 2 == 0 && CN == 4, "16-byte loads");
#pragma unroll 4
    for (int s = 0; s < S; ++s) {
        ulonglong2 av[RP / 2];
#pragma unroll
        for (int i = 0; i < RP / 2; ++i) av[i] = *reinterpret_cast<const ulonglong2*>(a + s * a_pitch + 4 * i);
        const float4 bv = *reinterpret_cast<const float4*>(b + s * b_pitch);
        const uint64_t bb[4] = {pack2(bv.x, bv.x), pack2(bv.y, bv.y), pack2(bv.z, bv.z), pack2(bv.w, bv.w)};
#pragma unroll
        for (int i = 0; i < RP; ++i)
#pragma unroll
            for (int j = 0; j < CN; ++j) acc[i][j] = ffma2(i & 1 ? av[i / 2].y : av[i / 2].x, bb[j], acc[i][j]);
    }
}

template <int RM, int CN>
__device__ __forceinline__ void zero2(uint64_t (&acc)[RM][CN])
{
#pragma unroll
    for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int j = 0; j < CN; ++j) acc[i][j] = 0ull;
}

// Logistic function from the approximate exponential and reciprocal (a few
// ulp; without the denormal handling of __expf and __fdividef, which changes
// nothing here: 1 + e^-x is never denormal, and e^-x is added to 1).
__device__ __forceinline__ float sigmoid_ftz(float x)
{
    float e, r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(x * -1.4426950408889634f));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + e));
    return r;
}

// Hidden activation and derivative. SiLU, the decoder's default, is inlined
// (one exponential and one divide for both); the others go through a call.
static __device__ __noinline__ float2 act_pair_any(int a, float x, float beta)
{
    return make_float2(act_fwd(a, x, beta), act_grad(a, x, beta));
}

__device__ __forceinline__ void act_pair(int a, float x, float beta, float& h, float& g)
{
    if (a == ATDF_ACT_SILU) {
        const float s = sigmoid_ftz(x);
        h = x * s;
        g = s * (1.0f + x * (1.0f - s));
    } else {
        const float2 v = act_pair_any(a, x, beta);
        h = v.x;
        g = v.y;
    }
}

static __device__ __noinline__ float act_any(int a, float x, float beta) { return act_fwd(a, x, beta); }

__device__ __forceinline__ float act_hidden(int a, float x, float beta)
{
    return a == ATDF_ACT_SILU ? x * sigmoid_ftz(x) : act_any(a, x, beta);
}

}  // namespace atdf
