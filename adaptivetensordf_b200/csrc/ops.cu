// Unfused drop-in operators of the projection path for sm_100a: the two
// indirect grid-sample ops, GradientCorrection's backward, the VM feature
// field, the decoder MLP, the X-ray line integral, node-error scoring and the
// MSE loss. They keep the reference's per-op interfaces so callers can swap
// them in one at a time; the fused leaf-major path lives in fused.cu.
//
// Reference: hyperacorn/csrc/modules/IndirectGridSample2D.cu:22-393,
// IndirectGridSample1D.cu:20-140, GradientCorrection.cu:22-48;
// hyperacorn/csrc/geometry/geometry_tensor_qo.cpp:257-380, Modules.h:23-149,
// geometry.cpp:33-53,176-253,977-1019.

#include <algorithm>

#include "atdf_common.cuh"

namespace atdf {

// V floats by one access.
template <int V>
struct Vec {
    float v[V];
};

template <int V>
__device__ __forceinline__ Vec<V> load_vec(const float* p)
{
    Vec<V> r;
    if constexpr (V == 4) {
        const float4 t = __ldg(reinterpret_cast<const float4*>(p));
        r.v[0] = t.x;
        r.v[1] = t.y;
        r.v[2] = t.z;
        r.v[3] = t.w;
    } else {
        r.v[0] = __ldg(p);
    }
    return r;
}

template <int V>
__device__ __forceinline__ void store_vec(float* p, const Vec<V>& r)
{
    if constexpr (V == 4)
        *reinterpret_cast<float4*>(p) = make_float4(r.v[0], r.v[1], r.v[2], r.v[3]);
    else
        *p = r.v[0];
}

// p[0..V) += w * r in global memory.
template <int V>
__device__ __forceinline__ void add_vec(float* p, float w, const Vec<V>& r)
{
    if constexpr (V == 4)
        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(__cvta_generic_to_global(p)),
                     "f"(__fmul_rn(w, r.v[0])), "f"(__fmul_rn(w, r.v[1])), "f"(__fmul_rn(w, r.v[2])),
                     "f"(__fmul_rn(w, r.v[3]))
                     : "memory");
    else
        atomicAdd(p, __fmul_rn(w, r.v[0]));
}

// ---------------------------------------------------------------------------
// grid sample 2D / 1D (one thread per sample, channels in a loop)
// ---------------------------------------------------------------------------
__global__ void gs2_fwd_kernel(const float* __restrict__ grid, int64_t N, int64_t C, int H, int W, int64_t sN,
                               int64_t sC, int64_t sH, int64_t sW, const int64_t* __restrict__ index,
                               const float* __restrict__ uv, int64_t S, float* __restrict__ out, int32_t* err)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= S) return;
    const int64_t n = index[i];
    if (n < 0 || n >= N) {
        set_err(err, ATDF_DEVERR_INDEX);
        for (int64_t c = 0; c < C; ++c) out[i * C + c] = 0.0f;
        return;
    }
    const Corner2 k = corners2(uv[2 * i], uv[2 * i + 1], H, W);
    const float* g = grid + n * sN;
    for (int64_t c = 0; c < C; ++c) {
        const float* gc = g + c * sC;
        out[i * C + c] = bilerp(k, gc[k.y0 * sH + k.x0 * sW], gc[k.y0 * sH + k.x1 * sW], gc[k.y1 * sH + k.x0 * sW],
                                gc[k.y1 * sH + k.x1 * sW]);
    }
}

// One channel's four terms each of the coordinate gradient's x and y chains, one
// rounding per operation (IndirectGridSample2D.cu:354-367).
__device__ __forceinline__ void coord_terms2(float vnw, float vne, float vsw, float vse, float ax0, float ax1, float ay0,
                                             float ay1, float go, float* tx, float* ty)
{
    tx[0] = __fmul_rn(__fmul_rn(__fmul_rn(-1.0f, vnw), ay1), go);
    tx[1] = __fmul_rn(__fmul_rn(vne, ay1), go);
    tx[2] = __fmul_rn(__fmul_rn(__fmul_rn(-1.0f, vsw), ay0), go);
    tx[3] = __fmul_rn(__fmul_rn(vse, ay0), go);
    ty[0] = __fmul_rn(__fmul_rn(__fmul_rn(-1.0f, vnw), ax1), go);
    ty[1] = __fmul_rn(__fmul_rn(__fmul_rn(-1.0f, vne), ax0), go);
    ty[2] = __fmul_rn(__fmul_rn(vsw, ax1), go);
    ty[3] = __fmul_rn(__fmul_rn(vse, ax0), go);
}

__global__ void gs2_bwd_kernel(const float* __restrict__ grid, int64_t N, int64_t C, int H, int W, int64_t sN,
                               int64_t sC, int64_t sH, int64_t sW, const int64_t* __restrict__ index,
                               const float* __restrict__ uv, int64_t S, const float* __restrict__ gout,
                               float* __restrict__ ggrid, float* __restrict__ guv, int32_t* err)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= S) return;
    const int64_t n = index[i];
    if (n < 0 || n >= N) {
        set_err(err, ATDF_DEVERR_INDEX);
        return;
    }
    const Corner2 k = corners2(uv[2 * i], uv[2 * i + 1], H, W);
    const float* g = grid + n * sN;
    float* gg = ggrid ? ggrid + n * C * H * W : nullptr;
    float gix = 0.0f, giy = 0.0f;
    const float ay1 = __fsub_rn(k.fy1, k.iy), ay0 = __fsub_rn(k.iy, k.fy0);
    const float ax1 = __fsub_rn(k.fx1, k.ix), ax0 = __fsub_rn(k.ix, k.fx0);
    for (int64_t c = 0; c < C; ++c) {
        const float go = gout[i * C + c];
        const float* gc = g + c * sC;
        if (gg) {
            float* ggc = gg + c * H * W;
            atomicAdd(&ggc[k.y0 * W + k.x0], __fmul_rn(k.w_nw, go));
            atomicAdd(&ggc[k.y0 * W + k.x1], __fmul_rn(k.w_ne, go));
            atomicAdd(&ggc[k.y1 * W + k.x0], __fmul_rn(k.w_sw, go));
            atomicAdd(&ggc[k.y1 * W + k.x1], __fmul_rn(k.w_se, go));
        }
        const float vnw = gc[k.y0 * sH + k.x0 * sW], vne = gc[k.y0 * sH + k.x1 * sW];
        const float vsw = gc[k.y1 * sH + k.x0 * sW], vse = gc[k.y1 * sH + k.x1 * sW];
        float tx[4], ty[4];
        coord_terms2(vnw, vne, vsw, vse, ax0, ax1, ay0, ay1, go, tx, ty);
        for (int j = 0; j < 4; ++j) {
            gix = __fadd_rn(gix, tx[j]);
            giy = __fadd_rn(giy, ty[j]);
        }
    }
    if (guv) {
        guv[2 * i] = __fadd_rn(guv[2 * i], __fdiv_rn(__fmul_rn(gix, (float)(W - 1)), 2.0f));
        guv[2 * i + 1] = __fadd_rn(guv[2 * i + 1], __fdiv_rn(__fmul_rn(giy, (float)(H - 1)), 2.0f));
    }
}

// Channels-last grids [N][H][W][C] with C a multiple of 4 and 16-byte aligned
// rows. Forward: a thread per sample and 4 channels.
__global__ void __launch_bounds__(256)
    gs2_fwd_cl_kernel(const float* __restrict__ grid, int64_t N, int C, int H, int W,
                      const int64_t* __restrict__ index, const float* __restrict__ uv, int64_t S,
                      float* __restrict__ out, int32_t* err)
{
    const int Q = C / 4;
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, i = e / Q;
    if (i >= S) return;
    const int c0 = (int)(e - i * Q) * 4;
    const int64_t n = index[i];
    Vec<4> r;
    if (n < 0 || n >= N) {
        set_err(err, ATDF_DEVERR_INDEX);
        for (int j = 0; j < 4; ++j) r.v[j] = 0.0f;
    } else {
        const Corner2 k = corners2(uv[2 * i], uv[2 * i + 1], H, W);
        const float* g = grid + n * (int64_t)H * W * C + c0;
        const Vec<4> nw = load_vec<4>(g + (int64_t)(k.y0 * W + k.x0) * C), ne = load_vec<4>(g + (int64_t)(k.y0 * W + k.x1) * C),
                     sw = load_vec<4>(g + (int64_t)(k.y1 * W + k.x0) * C), se = load_vec<4>(g + (int64_t)(k.y1 * W + k.x1) * C);
#pragma unroll
        for (int j = 0; j < 4; ++j) r.v[j] = bilerp(k, nw.v[j], ne.v[j], sw.v[j], se.v[j]);
    }
    store_vec<4>(out + e * 4, r);
}

// Adjoint into a channels-last gradient by 16-byte reductions. Q threads per
// sample (a power of two, 4 CQ channels each; Q = 1 for the channel counts
// that do not split so). The coordinate gradient is one chain of roundings over
// the channels in order (IndirectGridSample2D.cu:354-367): every thread forms
// the terms of its channels, then the chain passes from thread to thread.
template <int Q>
__global__ void __launch_bounds__(256)
    gs2_bwd_cl_kernel(const float* __restrict__ grid, int64_t N, int C, int H, int W,
                      const int64_t* __restrict__ index, const float* __restrict__ uv, int64_t S,
                      const float* __restrict__ gout, float* __restrict__ ggrid, float* __restrict__ guv, int32_t* err)
{
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t i = e / Q;
    const int q = (int)(e % Q);
    const int64_t n = i < S ? index[i] : -1;
    const bool ok = n >= 0 && n < N;
    if (i < S && !ok) set_err(err, ATDF_DEVERR_INDEX);
    const Corner2 k = corners2(ok ? uv[2 * i] : 0.0f, ok ? uv[2 * i + 1] : 0.0f, H, W);
    const int64_t base = (ok ? n : 0) * (int64_t)H * W * C;
    const int64_t o[4] = {base + (int64_t)(k.y0 * W + k.x0) * C, base + (int64_t)(k.y0 * W + k.x1) * C,
                          base + (int64_t)(k.y1 * W + k.x0) * C, base + (int64_t)(k.y1 * W + k.x1) * C};
    float gix = 0.0f, giy = 0.0f;
    const float ay1 = __fsub_rn(k.fy1, k.iy), ay0 = __fsub_rn(k.iy, k.fy0);
    const float ax1 = __fsub_rn(k.fx1, k.ix), ax0 = __fsub_rn(k.ix, k.fx0);
    // the Q threads take neighbouring groups of 4 channels, round by round
    for (int c0 = 0; c0 < C; c0 += 4 * Q) {
        const int c = c0 + 4 * q;
        float tx[16], ty[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) tx[j] = ty[j] = 0.0f;
        if (ok) {
            const Vec<4> go = load_vec<4>(gout + i * C + c);
            add_vec<4>(ggrid + o[0] + c, k.w_nw, go);
            add_vec<4>(ggrid + o[1] + c, k.w_ne, go);
            add_vec<4>(ggrid + o[2] + c, k.w_sw, go);
            add_vec<4>(ggrid + o[3] + c, k.w_se, go);
            const Vec<4> nw = load_vec<4>(grid + o[0] + c), ne = load_vec<4>(grid + o[1] + c),
                         sw = load_vec<4>(grid + o[2] + c), se = load_vec<4>(grid + o[3] + c);
#pragma unroll
            for (int j = 0; j < 4; ++j)
                coord_terms2(nw.v[j], ne.v[j], sw.v[j], se.v[j], ax0, ax1, ay0, ay1, go.v[j], tx + 4 * j, ty + 4 * j);
        }
#pragma unroll
        for (int r = 0; r < Q; ++r) {
            float sx = gix, sy = giy;
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                sx = __fadd_rn(sx, tx[j]);
                sy = __fadd_rn(sy, ty[j]);
            }
            gix = Q == 1 ? sx : __shfl_sync(0xffffffffu, sx, r, Q);
            giy = Q == 1 ? sy : __shfl_sync(0xffffffffu, sy, r, Q);
        }
    }
    if (!ok || q != 0) return;
    guv[2 * i] = __fadd_rn(guv[2 * i], __fdiv_rn(__fmul_rn(gix, (float)(W - 1)), 2.0f));
    guv[2 * i + 1] = __fadd_rn(guv[2 * i + 1], __fdiv_rn(__fmul_rn(giy, (float)(H - 1)), 2.0f));
}

// [N][C][HW] to [N][HW][C] or back, a block per 128 texels of one n: whole rows
// of either layout through shared memory.
constexpr int kLayoutTexels = 128;

__global__ void __launch_bounds__(256)
    grid_layout_kernel(const float* __restrict__ src, int C, int HW, bool to_cl, float* __restrict__ dst)
{
    extern __shared__ float s_tile[];  // [C][kLayoutTexels + 1]
    const int chunks = (HW + kLayoutTexels - 1) / kLayoutTexels;
    const int64_t base = (int64_t)(blockIdx.x / chunks) * C * HW;
    const int x0 = (int)(blockIdx.x % chunks) * kLayoutTexels, nx = min(kLayoutTexels, HW - x0);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    // channel rows by warps, texel rows as one run of nx * C values (c and x of
    // a thread's next value without a division)
    const int dc = blockDim.x % C, dx = blockDim.x / C;
    auto rows = [&](auto move) {
        for (int c = warp; c < C; c += warps)
#pragma unroll
            for (int x = lane; x < kLayoutTexels; x += 32)
                if (x < nx) move(c, x, base + (int64_t)c * HW + x0 + x);
    };
    auto texels = [&](auto move) {
        int c = threadIdx.x % C, x = threadIdx.x / C;
#pragma unroll 4
        for (int e = threadIdx.x; e < C * nx; e += blockDim.x) {
            move(c, x, base + (int64_t)x0 * C + e);
            c += dc;
            x += dx;
            if (c >= C) {
                c -= C;
                ++x;
            }
        }
    };
    auto in = [&](int c, int x, int64_t at) { s_tile[c * (kLayoutTexels + 1) + x] = __ldg(src + at); };
    auto out = [&](int c, int x, int64_t at) { dst[at] = s_tile[c * (kLayoutTexels + 1) + x]; };
    if (to_cl)
        rows(in);
    else
        texels(in);
    __syncthreads();
    if (to_cl)
        texels(out);
    else
        rows(out);
}

// V channels at a time: 16-byte stores when the channel count allows (V = 4).
template <int V>
__global__ void gs1_fwd_kernel(const float* __restrict__ grid, int64_t N, int64_t C, int W, int64_t sN, int64_t sC,
                               int64_t sW, const int64_t* __restrict__ index, const float* __restrict__ uv, int64_t S,
                               float* __restrict__ out, int32_t* err)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= S) return;
    const int64_t n = index[i];
    const bool ok = n >= 0 && n < N;
    if (!ok) set_err(err, ATDF_DEVERR_INDEX);
    const Corner1 k = corners1(uv[i], W);
    const float* g = grid + (ok ? n * sN : 0);
    for (int64_t c = 0; c < C; c += V) {
        Vec<V> r;
#pragma unroll
        for (int j = 0; j < V; ++j)
            r.v[j] = ok ? lerp1(k, g[(c + j) * sC + k.x0 * sW], g[(c + j) * sC + k.x1 * sW]) : 0.0f;
        store_vec<V>(out + i * C + c, r);
    }
}

// SMEM_SUM: the grid's gradient fits in shared memory. Many samples add to
// few entries, so each block sums its own copy there and adds it once;
// larger grids take global atomics.
template <bool SMEM_SUM>
__global__ void __launch_bounds__(256)
    gs1_bwd_kernel(const float* __restrict__ grid, int64_t N, int64_t C, int W, int64_t sN, int64_t sC, int64_t sW,
                   const int64_t* __restrict__ index, const float* __restrict__ uv, int64_t S,
                   const float* __restrict__ gout, float* __restrict__ ggrid, float* __restrict__ guv, int32_t* err)
{
    extern __shared__ float s_sum[];
    const int64_t total = N * C * W;
    if (SMEM_SUM) {
        for (int64_t j = threadIdx.x; j < total; j += blockDim.x) s_sum[j] = 0.0f;
        __syncthreads();
    }
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < S; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t n = index[i];
        if (n < 0 || n >= N) {
            set_err(err, ATDF_DEVERR_INDEX);
            continue;
        }
        const Corner1 k = corners1(uv[i], W);
        const float* g = grid + n * sN;
        float* gg = SMEM_SUM ? s_sum + n * C * W : ggrid ? ggrid + n * C * W : nullptr;
        float gix = 0.0f;
        const float a1 = __fsub_rn(k.fx1, k.ix), a0 = __fsub_rn(k.ix, k.fx0);
        for (int64_t c = 0; c < C; ++c) {
            const float go = gout[i * C + c];
            if (gg) {
                atomicAdd(&gg[c * W + k.x0], __fmul_rn(k.w0, go));
                atomicAdd(&gg[c * W + k.x1], __fmul_rn(k.w1, go));
            }
            const float v0 = g[c * sC + k.x0 * sW], v1 = g[c * sC + k.x1 * sW];
            gix = __fadd_rn(gix, __fmul_rn(__fmul_rn(__fmul_rn(-1.0f, v0), a1), go));
            gix = __fadd_rn(gix, __fmul_rn(__fmul_rn(v1, a0), go));
        }
        if (guv) guv[i] = __fadd_rn(guv[i], __fdiv_rn(__fmul_rn(gix, (float)(W - 1)), 2.0f));
    }
    if (!SMEM_SUM) return;
    __syncthreads();
    for (int64_t j = threadIdx.x; j < total; j += blockDim.x) {
        const float v = s_sum[j];
        if (v != 0.0f) atomicAdd(&ggrid[j], v);
    }
}

// The 1D adjoint with 16-byte reductions into one of `copies` channels-last
// copies of the gradient ([copy][n][W][C], zeroed): a few hundred entries take
// every sample, so one copy would serialise them, and shared-memory float adds
// (a compare-and-swap loop) took 146 us for 1 M samples of 16 channels.
__global__ void __launch_bounds__(256)
    gs1_bwd_copies_kernel(const float* __restrict__ grid, int64_t N, int C, int W, int64_t sN, int64_t sC, int64_t sW,
                          const int64_t* __restrict__ index, const float* __restrict__ uv, int64_t S,
                          const float* __restrict__ gout, float* __restrict__ rep, int copies,
                          float* __restrict__ guv, int32_t* err)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= S) return;
    const int64_t n = index[i];
    if (n < 0 || n >= N) {
        set_err(err, ATDF_DEVERR_INDEX);
        return;
    }
    const Corner1 k = corners1(uv[i], W);
    const float* g = grid + n * sN;
    float* r0 = rep + (((int64_t)(blockIdx.x % copies) * N + n) * W + k.x0) * C;
    float* r1 = rep + (((int64_t)(blockIdx.x % copies) * N + n) * W + k.x1) * C;
    float gix = 0.0f;
    const float a1 = __fsub_rn(k.fx1, k.ix), a0 = __fsub_rn(k.ix, k.fx0);
    for (int c = 0; c < C; c += 4) {
        const Vec<4> go = load_vec<4>(gout + i * C + c);
        add_vec<4>(r0 + c, k.w0, go);
        add_vec<4>(r1 + c, k.w1, go);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float v0 = g[(c + j) * sC + k.x0 * sW], v1 = g[(c + j) * sC + k.x1 * sW];
            gix = __fadd_rn(gix, __fmul_rn(__fmul_rn(__fmul_rn(-1.0f, v0), a1), go.v[j]));
            gix = __fadd_rn(gix, __fmul_rn(__fmul_rn(v1, a0), go.v[j]));
        }
    }
    guv[i] = __fadd_rn(guv[i], __fdiv_rn(__fmul_rn(gix, (float)(W - 1)), 2.0f));
}

// ggrid [N][C][W] += the sum of the copies (in FP64, one rounding).
__global__ void gs1_sum_copies_kernel(const float* __restrict__ rep, int copies, int64_t N, int C, int W,
                                      float* __restrict__ ggrid)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, total = N * C * W;
    if (i >= total) return;
    double acc = 0.0;
    for (int r = 0; r < copies; ++r) acc += (double)rep[r * total + i];
    const int64_t n = i / ((int64_t)W * C);
    const int x = (int)(i / C % W), c = (int)(i % C);
    ggrid[(n * C + c) * W + x] += (float)acc;
}

__global__ void gradcorr_bwd_kernel(const float* __restrict__ dir, const int64_t* __restrict__ ray, int64_t R,
                                    const float* __restrict__ gin, int64_t S, float* __restrict__ gout, int32_t* err)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= S) return;
    const int64_t r = ray[i];
    if (r < 0 || r >= R) {
        set_err(err, ATDF_DEVERR_INDEX);
        return;
    }
    const float d0 = dir[3 * r], d1 = dir[3 * r + 1], d2 = dir[3 * r + 2];
    const float g0 = gin[3 * i], g1 = gin[3 * i + 1], g2 = gin[3 * i + 2];
    // grad - grad.dot(direction) * direction, one rounding per operation
    // (the dot product summed left to right), so the result is reproducible
    const float dot = __fadd_rn(__fadd_rn(__fmul_rn(g0, d0), __fmul_rn(g1, d1)), __fmul_rn(g2, d2));
    gout[3 * i] = __fsub_rn(g0, __fmul_rn(dot, d0));
    gout[3 * i + 1] = __fsub_rn(g1, __fmul_rn(dot, d1));
    gout[3 * i + 2] = __fsub_rn(g2, __fmul_rn(dot, d2));
}

// ---------------------------------------------------------------------------
// VM feature field, FP32, channels-last. A thread takes N pieces of V channels
// of one sample (V = 4 with 16-byte accesses when the channel count and the
// pointers allow it, else 1; N = 2 for channel counts that are multiples of 8,
// which halves the threads that repeat a sample's geometry). Neighbouring
// threads read and write neighbouring pieces: one thread per sample walking
// its channels left every access of a warp in a cache line of its own.
// ---------------------------------------------------------------------------
// Slot and coordinates of sample i; slot -1 (zero features) for a bad index
// (which sets the error bit) and outside the ROI.
__device__ __forceinline__ int64_t vm_sample(const atdf_field_t& f, const float* __restrict__ pmin,
                                             const float* __restrict__ pmax, int64_t num_nodes,
                                             const float* __restrict__ pos, const int64_t* __restrict__ node,
                                             int64_t i, SampleGeo& g, int32_t* err)
{
    const int64_t nd = node[i];
    if (nd < 0 || nd >= num_nodes) {
        set_err(err, ATDF_DEVERR_INDEX);
        return -1;
    }
    const int64_t slot = f.leaf_slot[nd];
    if (slot < 0 || slot >= f.num_slots) {
        if (slot >= f.num_slots) set_err(err, ATDF_DEVERR_INDEX);
        return -1;
    }
    const float p[3] = {pos[3 * i], pos[3 * i + 1], pos[3 * i + 2]};
    g = sample_geo(p, pmin + 3 * nd, pmax + 3 * nd, f.roi_min, f.roi_max);
    return slot;
}

// Bilinear value of plane m (P: the slot's plane) and linear value of line m.
template <int V>
__device__ __forceinline__ void vm_values(const Corner2& k, const Corner1& l, const float* P, const float* L, int W,
                                          int C, int c0, Vec<V>& mat, Vec<V>& vec)
{
    const Vec<V> nw = load_vec<V>(P + (k.y0 * W + k.x0) * C + c0), ne = load_vec<V>(P + (k.y0 * W + k.x1) * C + c0),
                 sw = load_vec<V>(P + (k.y1 * W + k.x0) * C + c0), se = load_vec<V>(P + (k.y1 * W + k.x1) * C + c0),
                 v0 = load_vec<V>(L + l.x0 * C + c0), v1 = load_vec<V>(L + l.x1 * C + c0);
#pragma unroll
    for (int i = 0; i < V; ++i) {
        mat.v[i] = bilerp(k, nw.v[i], ne.v[i], sw.v[i], se.v[i]);
        vec.v[i] = lerp1(l, v0.v[i], v1.v[i]);
    }
}

template <int V, int N>
__global__ void __launch_bounds__(256)
    vm_fwd_kernel(atdf_field_t f, const float* __restrict__ pmin, const float* __restrict__ pmax, int64_t num_nodes,
                  const float* __restrict__ pos, const int64_t* __restrict__ node, int64_t S, float* __restrict__ out,
                  int32_t* err)
{
    const int C = f.channels, Q = C / (V * N);
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t i = e / Q;
    if (i >= S) return;
    const int c0 = (int)(e - i * Q) * V;  // channels c0 + n Q V .. + V - 1 of piece n
    float* o = out + i * (f.mode ? 3 * C : C) + c0;
    SampleGeo g;
    const int64_t slot = vm_sample(f, pmin, pmax, num_nodes, pos, node, i, g, err);
    Vec<V> acc[N];
#pragma unroll
    for (int n = 0; n < N; ++n)
#pragma unroll
        for (int j = 0; j < V; ++j) acc[n].v[j] = 0.0f;
    if (slot >= 0) {
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            const int H = f.plane_h[m], W = f.plane_w[m];
            const Corner2 k = corners2(g.pu[m], g.pv[m], H, W);
            const Corner1 l = corners1(g.lu[m], f.line_len[m]);
            const float* P = (const float*)f.plane[m] + slot * (int64_t)H * W * C;
#pragma unroll
            for (int n = 0; n < N; ++n) {
                Vec<V> mat, vec;
                vm_values<V>(k, l, P, (const float*)f.line[m], W, C, c0 + n * Q * V, mat, vec);
#pragma unroll
                for (int j = 0; j < V; ++j) {
                    const float prod = __fmul_rn(mat.v[j], vec.v[j]);
                    acc[n].v[j] = m == 0 || f.mode ? prod : __fadd_rn(acc[n].v[j], prod);
                }
                if (f.mode) store_vec<V>(o + m * C + n * Q * V, acc[n]);
            }
        }
    } else if (f.mode) {
        for (int m = 0; m < 3; ++m)
            for (int n = 0; n < N; ++n) store_vec<V>(o + m * C + n * Q * V, acc[n]);
    }
    if (!f.mode)
#pragma unroll
        for (int n = 0; n < N; ++n) store_vec<V>(o + n * Q * V, acc[n]);
}

// The adjoint: plane gradients by (vector) reductions into global memory.
// Line gradients collect every sample in a few hundred entries, so with
// smem_lines each block sums its own copy in shared memory (the blocks stride
// over the samples) and adds it once; more entries than fit go to global
// memory directly. One piece of channels a thread: two put twice as many
// samples in a warp, whose adds to the shared lines then collide more (98 us
// against 169 us for 290 k samples of 8 channels; one thread a sample with
// global line atomics took 1942 us).
template <int V>
__global__ void __launch_bounds__(256)
    vm_bwd_kernel(atdf_field_t f, const float* __restrict__ pmin, const float* __restrict__ pmax, int64_t num_nodes,
                  const float* __restrict__ pos, const int64_t* __restrict__ node, int64_t S,
                  const float* __restrict__ gout, atdf_field_grad_t gr, bool smem_lines, int32_t* err)
{
    extern __shared__ __align__(16) float s_line[];
    const int C = f.channels, Q = C / V;
    const int off[4] = {0, f.line_len[0] * C, (f.line_len[0] + f.line_len[1]) * C,
                        (f.line_len[0] + f.line_len[1] + f.line_len[2]) * C};
    const int lane = threadIdx.x & 31;
    const bool pow2_q = smem_lines && Q < 32 && (Q & (Q - 1)) == 0;
    if (smem_lines) {
        for (int i = threadIdx.x; i < off[3]; i += blockDim.x) s_line[i] = 0.0f;
        __syncthreads();
    }
    // the loop bounds are the block's, so that all lanes of a warp reach the votes and shuffles
    for (int64_t e0 = (int64_t)blockIdx.x * blockDim.x; e0 < S * Q; e0 += (int64_t)gridDim.x * blockDim.x) {
        const int64_t e = e0 + threadIdx.x, i = e / Q;
        const int c0 = (int)(e - i * Q) * V;
        SampleGeo g;
        int64_t slot = -1;
        if (e < S * Q) {
            const int64_t nd = node[i];
            if (nd < 0 || nd >= num_nodes)
                set_err(err, ATDF_DEVERR_INDEX);
            else
                slot = vm_sample(f, pmin, pmax, num_nodes, pos, node, i, g, nullptr);
        }
        // The samples of a ray follow one another: where a whole warp falls
        // between the same two entries of a line (the y line under a beam
        // normal to y) its shared-memory adds would all collide.
        bool same[3] = {false, false, false};
        const bool whole = pow2_q && __all_sync(0xffffffffu, slot >= 0);
        if (whole) {
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                const Corner1 l = corners1(g.lu[m], f.line_len[m]);
                const int x0 = __shfl_sync(0xffffffffu, l.x0, 0), x1 = __shfl_sync(0xffffffffu, l.x1, 0);
                same[m] = __all_sync(0xffffffffu, l.x0 == x0 && l.x1 == x1);
            }
        }
        if (slot < 0) continue;
        const float* go = gout + i * (f.mode ? 3 * C : C);
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            const int H = f.plane_h[m], W = f.plane_w[m];
            const Corner2 k = corners2(g.pu[m], g.pv[m], H, W);
            const Corner1 l = corners1(g.lu[m], f.line_len[m]);
            const int64_t base = slot * (int64_t)H * W * C;
            Vec<V> mat, vec;
            vm_values<V>(k, l, (const float*)f.plane[m] + base, (const float*)f.line[m], W, C, c0, mat, vec);
            const Vec<V> gf = load_vec<V>(go + (f.mode ? m * C : 0) + c0);
            Vec<V> gm, gv;
#pragma unroll
            for (int j = 0; j < V; ++j) {
                gm.v[j] = __fmul_rn(gf.v[j], vec.v[j]);
                gv.v[j] = __fmul_rn(gf.v[j], mat.v[j]);
            }
            if (gr.plane[m]) {
                float* GP = gr.plane[m] + base + c0;
                add_vec<V>(GP + (k.y0 * W + k.x0) * C, k.w_nw, gm);
                add_vec<V>(GP + (k.y0 * W + k.x1) * C, k.w_ne, gm);
                add_vec<V>(GP + (k.y1 * W + k.x0) * C, k.w_sw, gm);
                add_vec<V>(GP + (k.y1 * W + k.x1) * C, k.w_se, gm);
            }
            if (!gr.line[m]) continue;
            if (smem_lines) {
                float* dst = s_line + off[m] + c0;
                if (same[m]) {  // one entry pair for the whole warp: its sums, added by one sample's lanes
#pragma unroll
                    for (int j = 0; j < V; ++j) {
                        float a0 = __fmul_rn(l.w0, gv.v[j]), a1 = __fmul_rn(l.w1, gv.v[j]);
                        for (int d = Q; d < 32; d <<= 1) {
                            a0 += __shfl_xor_sync(0xffffffffu, a0, d);
                            a1 += __shfl_xor_sync(0xffffffffu, a1, d);
                        }
                        if (lane < Q) {
                            atomicAdd(&dst[l.x0 * C + j], a0);
                            atomicAdd(&dst[l.x1 * C + j], a1);
                        }
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < V; ++j) {
                        atomicAdd(&dst[l.x0 * C + j], __fmul_rn(l.w0, gv.v[j]));
                        atomicAdd(&dst[l.x1 * C + j], __fmul_rn(l.w1, gv.v[j]));
                    }
                }
            } else {
                add_vec<V>(gr.line[m] + l.x0 * C + c0, l.w0, gv);
                add_vec<V>(gr.line[m] + l.x1 * C + c0, l.w1, gv);
            }
        }
    }
    if (!smem_lines) return;
    __syncthreads();
    for (int m = 0; m < 3; ++m)
        if (gr.line[m])
            for (int i = threadIdx.x; i < f.line_len[m] * C; i += blockDim.x) {
                const float v = s_line[off[m] + i];
                if (v != 0.0f) atomicAdd(&gr.line[m][i], v);
            }
}

// ---------------------------------------------------------------------------
// line integral, node-error scoring, MSE loss
// ---------------------------------------------------------------------------
__global__ void integrate_kernel(const float* __restrict__ vals, const float* __restrict__ w,
                                 const int64_t* __restrict__ ray, int64_t S, int C, int64_t R, float* img,
                                 int32_t* err)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= S) return;
    const int64_t r = ray[i];
    if (r < 0 || r >= R) {
        set_err(err, ATDF_DEVERR_INDEX);
        return;
    }
    const float wi = w[i];
    for (int c = 0; c < C; ++c) atomicAdd(&img[c * R + r], __fmul_rn(vals[i * C + c], wi));
}

__global__ void node_loss_kernel(const float* __restrict__ prl, int C, int64_t R, const int64_t* __restrict__ ray,
                                 const int64_t* __restrict__ node, const float* __restrict__ w, int64_t S,
                                 int64_t num_nodes, double* ls, double* ws, int32_t* err)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= S) return;
    const int64_t r = ray[i], nd = node[i];
    if (r < 0 || r >= R || nd < 0 || nd >= num_nodes) {
        set_err(err, ATDF_DEVERR_INDEX);
        return;
    }
    double l = 0.0;
    for (int c = 0; c < C; ++c) l += (double)prl[c * R + r];
    l /= (double)C;
    const double wi = (double)w[i];
    atomicAdd(&ls[nd], l * wi);
    atomicAdd(&ws[nd], wi);
}

__global__ void mse_kernel(const float* __restrict__ img, const float* __restrict__ tgt, int64_t n, float scale,
                           double* loss, float* __restrict__ gimg, float* __restrict__ prl)
{
    __shared__ double red[256];
    double acc = 0.0;
    const float gs = scale * 2.0f / (float)n;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float d = img[i] - tgt[i];
        acc += (double)d * (double)d;
        if (gimg) gimg[i] = gs * d;
        if (prl) prl[i] = d * d;
    }
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
        if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0 && loss) atomicAdd(loss, red[0] * (double)scale / (double)n);
}

}  // namespace atdf

using namespace atdf;

static inline unsigned blocks_for(int64_t n, int t = 256) { return (unsigned)div_up(n, t); }

extern "C" {

// Strides of a dense channels-last grid that 16-byte accesses can take.
static bool channels_last4(const float* grid, int64_t C, int64_t H, int64_t W, const int64_t* s)
{
    return C % 4 == 0 && (reinterpret_cast<uintptr_t>(grid) & 15) == 0 && s[1] == 1 && s[3] == C && s[2] == C * W &&
           s[0] == C * W * H && C <= INT32_MAX / 4;
}

int atdf_grid_sample2d_forward(const float* grid, int64_t N, int64_t C, int64_t H, int64_t W,
                               const int64_t* s, const int64_t* index, const float* uv, int64_t S, float* out,
                               int32_t* dev_error, atdf_stream_t stream)
{
    if (!grid || !s || N <= 0 || C <= 0 || H <= 0 || W <= 0 || S < 0 || (S > 0 && (!index || !uv || !out)))
        return ATDF_ERR_INVALID_ARGUMENT;
    if (S == 0) return ATDF_OK;
    if (channels_last4(grid, C, H, W, s) && (reinterpret_cast<uintptr_t>(out) & 15) == 0)
        gs2_fwd_cl_kernel<<<blocks_for(S * (C / 4)), 256, 0, (cudaStream_t)stream>>>(grid, N, (int)C, (int)H, (int)W,
                                                                                     index, uv, S, out, dev_error);
    else
        gs2_fwd_kernel<<<blocks_for(S), 256, 0, (cudaStream_t)stream>>>(grid, N, C, (int)H, (int)W, s[0], s[1], s[2],
                                                                        s[3], index, uv, S, out, dev_error);
    ATDF_LAUNCH_CHECK();
    return ATDF_OK;
}

int atdf_grid_sample2d_backward(const float* grid, int64_t N, int64_t C, int64_t H, int64_t W, const int64_t* s,
                                const int64_t* index, const float* uv, int64_t S, const float* grad_out,
                                float* grad_grid, float* grad_uv, int32_t* dev_error, atdf_stream_t stream)
{
    if (!grid || !s || N <= 0 || C <= 0 || H <= 0 || W <= 0 || S < 0 || (S > 0 && (!index || !uv || !grad_out)))
        return ATDF_ERR_INVALID_ARGUMENT;
    if (S == 0) return ATDF_OK;
    gs2_bwd_kernel<<<blocks_for(S), 256, 0, (cudaStream_t)stream>>>(grid, N, C, (int)H, (int)W, s[0], s[1], s[2],
                                                                    s[3], index, uv, S, grad_out, grad_grid, grad_uv,
                                                                    dev_error);
    ATDF_LAUNCH_CHECK();
    return ATDF_OK;
}

int atdf_grid_sample2d_backward_channels_last(const float* grid, int64_t N, int64_t C, int64_t H, int64_t W,
                                              const int64_t* index, const float* uv, int64_t S, const float* grad_out,
                                              float* grad_grid, float* grad_uv, int32_t* dev_error,
                                              atdf_stream_t stream)
{
    if (!grid || !grad_grid || !grad_uv || N <= 0 || C <= 0 || H <= 0 || W <= 0 || S < 0 ||
        (S > 0 && (!index || !uv || !grad_out)))
        return ATDF_ERR_INVALID_ARGUMENT;
    if (C % 4 != 0 || ((reinterpret_cast<uintptr_t>(grid) | reinterpret_cast<uintptr_t>(grad_grid) |
                        reinterpret_cast<uintptr_t>(grad_out)) & 15) != 0)
        return ATDF_ERR_UNSUPPORTED;
    if (S == 0) return ATDF_OK;
    const int q = C % 32 == 0 ? 8 : C % 16 == 0 ? 4 : C % 8 == 0 ? 2 : 1;
    auto kernel = q == 8 ? gs2_bwd_cl_kernel<8> : q == 4 ? gs2_bwd_cl_kernel<4> : q == 2 ? gs2_bwd_cl_kernel<2>
                                                                                     : gs2_bwd_cl_kernel<1>;
    kernel<<<blocks_for(S * q), 256, 0, (cudaStream_t)stream>>>(grid, N, (int)C, (int)H, (int)W, index, uv, S, grad_out,
                                                                grad_grid, grad_uv, dev_error);
    ATDF_LAUNCH_CHECK();
    return ATDF_OK;
}

int atdf_grid_layout(const float* src, int64_t N, int64_t C, int64_t HW, int32_t to_channels_last, float* dst,
                     atdf_stream_t stream)
{
    if (N < 0 || C <= 0 || HW <= 0 || (N > 0 && (!src || !dst))) return ATDF_ERR_INVALID_ARGUMENT;
    const int64_t smem = C * (kLayoutTexels + 1) * 4, blocks = N * div_up(HW, kLayoutTexels);
    if (smem > 48 * 1024 || blocks > INT32_MAX || C * HW > INT32_MAX) return ATDF_ERR_UNSUPPORTED;
    if (N == 0) return ATDF_OK;
    grid_layout_kernel<<<(unsigned)blocks, 256, smem, (cudaStream_t)stream>>>(src, (int)C, (int)HW,
                                                                             to_channels_last != 0, dst);
    ATDF_LAUNCH_CHECK();
    return ATDF_OK;
}

int atdf_grid_sample1d_forward(const float* grid, int64_t N, int64_t C, int64_t W, const int64_t* s,
                               const int64_t* index, const float* uv, int64_t S, float* out, int32_t* dev_error,
                               atdf_stream_t stream)
{
    if (!grid || !s || N <= 0 || C <= 0 || W <= 0 || S < 0 || (S > 0 && (!index || !uv || !out)))
        return ATDF_ERR_INVALID_ARGUMENT;
    if (S == 0) return ATDF_OK;
    const bool vec = C % 4 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
    (vec ? gs1_fwd_kernel<4> : gs1_fwd_kernel<1>)<<<blocks_for(S), 256, 0, (cudaStream_t)stream>>>(
        grid, N, C, (int)W, s[0], s[1], s[2], index, uv, S, out, dev_error);
    ATDF_LAUNCH_CHECK();
    return ATDF_OK;
}

int atdf_grid_sample1d_backward(const float* grid, int64_t N, int64_t C, int64_t W, const int64_t* s,
                                const int64_t* index, const float* uv, int64_t S, const float* grad_out,
                                float* grad_grid, float* grad_uv, int32_t* dev_error, atdf_stream_t stream)
{
    if (!grid || !s || N <= 0 || C <= 0 || W <= 0 || S < 0 || (S > 0 && (!index || !uv || !grad_out)))
        return ATDF_ERR_INVALID_ARGUMENT;
    if (S == 0) return ATDF_OK;
    // a block's copy of the gradient: up to 64 KB, so that three blocks share an
    // SM, and enough samples to repay clearing and adding it: 16 channels, global
    // and shared, 17 entries, 1000 samples 10 and 21 us, 4000: 19 and 21, 16000: 72
    // and 23; 1000 entries, 4000 samples 12 and 16, 20000: 15 and 17, 64000: 38 and 19
    const bool smem_sum = grad_grid && N * C * W * 4 <= 64 * 1024 && S >= std::max<int64_t>(4096, 24 * N * W);
    const size_t smem = smem_sum ? (size_t)(N * C * W * 4) : 0;
    auto kernel = smem_sum ? gs1_bwd_kernel<true> : gs1_bwd_kernel<false>;
    unsigned blocks = blocks_for(S);
    if (smem_sum) {
        int dev = 0, sms = 0, per = 0;
        if (const int e = allow_dynamic_shared((const void*)kernel, (int)smem)) return e;
        ATDF_CUDA_TRY(cudaGetDevice(&dev));
        ATDF_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        ATDF_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, (const void*)kernel, 256, smem));
        if (per > 0 && blocks > (unsigned)(sms * per)) blocks = (unsigned)(sms * per);
    }
    kernel<<<blocks, 256, smem, (cudaStream_t)stream>>>(grid, N, C, (int)W, s[0], s[1], s[2], index, uv, S, grad_out,
                                                        grad_grid, grad_uv, dev_error);
    ATDF_LAUNCH_CHECK();
    return ATDF_OK;
}

int atdf_grid_sample1d_backward_copies(const float* grid, int64_t N, int64_t C, int64_t W, const int64_t* s,
                                       const int64_t* index, const float* uv, int64_t S, const float* grad_out,
                                       float* grad_grid, float* grad_uv, float* scratch, int32_t copies,
                                       int32_t* dev_error, atdf_stream_t stream)
{
    if (!grid || !s || !grad_grid || !grad_uv || !scratch || copies <= 0 || N <= 0 || C <= 0 || W <= 0 || S < 0 ||
        (S > 0 && (!index || !uv || !grad_out)))
        return ATDF_ERR_INVALID_ARGUMENT;
    if (C % 4 != 0 || C > INT32_MAX / 4 || W > INT32_MAX || N * C * W > INT32_MAX ||
        ((reinterpret_cast<uintptr_t>(grad_out) | reinterpret_cast<uintptr_t>(scratch)) & 15) != 0)
        return ATDF_ERR_UNSUPPORTED;
    if (S == 0) return ATDF_OK;
    const cudaStream_t st = (cudaStream_t)stream;
    ATDF_CUDA_TRY(cudaMemsetAsync(scratch, 0, (size_t)copies * N * C * W * 4, st));
    gs1_bwd_copies_kernel<<<blocks_for(S), 256, 0, st>>>(grid, N, (int)C, (int)W, s[0], s[1], s[2], index, uv, S,
                                                         grad_out, scratch, copies, grad_uv, dev_error);
    ATDF_LAUNCH_CHECK();
    gs1_sum_copies_kernel<<<blocks_for(N * C * W), 256, 0, st>>>(scratch, copies, N, (int)C, (int)W, grad_grid);
    ATDF_LAUNCH_CHECK();
    return ATDF_OK;
}

int atdf_gradient_correction_backward(const float* ray_direction, const int64_t* ray_index, int64_t num_rays,
                                      const float* grad_in, int64_t S, float* grad_out, int32_t* dev_error,
                                      atdf_stream_t stream)
{
    if (S < 0 || (S > 0 && (!ray_direction || !ray_index || !grad_in || !grad_out))) return ATDF_ERR_INVALID_ARGUMENT;
    if (S == 0) return ATDF_OK;
    gradcorr_bwd_kernel<<<blocks_for(S), 256, 0, (cudaStream_t)stream>>>(ray_direction, ray_index, num_rays, grad_in,
                                                                         S, grad_out, dev_error);
    ATDF_LAUNCH_CHECK();
    return ATDF_OK;
}

static bool field_ok(const atdf_field_t* f)
{
    if (!f || f->channels <= 0 || (f->mode != 0 && f->mode != 1) || !f->leaf_slot) return false;
    for (int m = 0; m < 3; ++m)
        if (!f->plane[m] || !f->line[m] || f->plane_h[m] <= 0 || f->plane_w[m] <= 0 || f->line_len[m] <= 0)
            return false;
    return true;
}

// Channels per thread: 8 or 4 by 16-byte accesses when the channel count is a
// multiple and every pointer is aligned, else 1.
static int vm_channels(const atdf_field_t* f, const float* features, const atdf_field_grad_t* g)
{
    uintptr_t bits = reinterpret_cast<uintptr_t>(features);
    for (int m = 0; m < 3; ++m) {
        bits |= reinterpret_cast<uintptr_t>(f->plane[m]) | reinterpret_cast<uintptr_t>(f->line[m]);
        if (g) bits |= reinterpret_cast<uintptr_t>(g->plane[m]) | reinterpret_cast<uintptr_t>(g->line[m]);
    }
    if ((bits & 15) != 0 || f->channels % 4 != 0) return 1;
    return f->channels % 8 == 0 ? 8 : 4;
}

int atdf_vm_features_forward(const atdf_field_t* field, const float* pmin, const float* pmax, int64_t num_nodes,
                             const float* position, const int64_t* node_id, int64_t S, float* out, int32_t* dev_error,
                             atdf_stream_t stream)
{
    if (!field_ok(field) || !pmin || !pmax || S < 0 || (S > 0 && (!position || !node_id || !out)))
        return ATDF_ERR_INVALID_ARGUMENT;
    if (field->dtype != ATDF_F32) return ATDF_ERR_UNSUPPORTED;
    if (S == 0) return ATDF_OK;
    const int per = vm_channels(field, out, nullptr);
    const int64_t threads = S * (field->channels / per);
    (per == 8 ? vm_fwd_kernel<4, 2> : per == 4 ? vm_fwd_kernel<4, 1> : vm_fwd_kernel<1, 1>)<<<blocks_for(threads), 256, 0, (cudaStream_t)stream>>>(
        *field, pmin, pmax, num_nodes, position, node_id, S, out, dev_error);
    ATDF_LAUNCH_CHECK();
    return ATDF_OK;
}

int atdf_vm_features_backward(const atdf_field_t* field, const float* pmin, const float* pmax, int64_t num_nodes,
                              const float* position, const int64_t* node_id, int64_t S, const float* grad_features,
                              const atdf_field_grad_t* grad, int32_t* dev_error, atdf_stream_t stream)
{
    if (!field_ok(field) || !pmin || !pmax || !grad || S < 0 || (S > 0 && (!position || !node_id || !grad_features)))
        return ATDF_ERR_INVALID_ARGUMENT;
    if (field->dtype != ATDF_F32) return ATDF_ERR_UNSUPPORTED;
    if (S == 0) return ATDF_OK;
    const int chan = std::min(4, vm_channels(field, grad_features, grad));
    const int64_t threads = S * (field->channels / chan);
    // a copy of the lines per block while two blocks of 256 threads still fit an SM
    const int64_t line_bytes =
        ((int64_t)field->line_len[0] + field->line_len[1] + field->line_len[2]) * field->channels * 4;
    const bool smem_lines = line_bytes <= 100 * 1024;
    auto kernel = chan == 4 ? vm_bwd_kernel<4> : vm_bwd_kernel<1>;
    const int smem = smem_lines ? (int)line_bytes : 0;
    unsigned blocks = blocks_for(threads);
    if (smem_lines) {
        if (const int e = allow_dynamic_shared((const void*)kernel, smem)) return e;
        int dev = 0, sms = 0, per = 0;
        ATDF_CUDA_TRY(cudaGetDevice(&dev));
        ATDF_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        ATDF_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, (const void*)kernel, 256, smem));
        if (per > 0 && blocks > (unsigned)(sms * per)) blocks = (unsigned)(sms * per);
    }
    kernel<<<blocks, 256, smem, (cudaStream_t)stream>>>(*field, pmin, pmax, num_nodes, position, node_id, S,
                                                        grad_features, *grad, smem_lines, dev_error);
    ATDF_LAUNCH_CHECK();
    return ATDF_OK;
}

int atdf_integrate_xray(const float* values, const float* weight, const int64_t* ray_index, int64_t S,
                        int32_t channels, int64_t num_rays, float* image, int32_t* dev_error, atdf_stream_t stream)
{
    if (S < 0 || channels <= 0 || num_rays < 0 || (S > 0 && (!values || !weight || !ray_index || !image)))
        return ATDF_ERR_INVALID_ARGUMENT;
    if (S == 0) return ATDF_OK;
    integrate_kernel<<<blocks_for(S), 256, 0, (cudaStream_t)stream>>>(values, weight, ray_index, S, channels, num_rays,
                                                                      image, dev_error);
    ATDF_LAUNCH_CHECK();
    return ATDF_OK;
}

int atdf_accumulate_loss_per_node(const float* per_ray_loss, int32_t channels, int64_t num_rays,
                                  const int64_t* ray_index, const int64_t* node_id, const float* weight, int64_t S,
                                  int64_t num_nodes, double* loss_sum, double* weight_sum, int32_t* dev_error,
                                  atdf_stream_t stream)
{
    if (S < 0 || channels <= 0 || !loss_sum || !weight_sum ||
        (S > 0 && (!per_ray_loss || !ray_index || !node_id || !weight)))
        return ATDF_ERR_INVALID_ARGUMENT;
    if (S == 0) return ATDF_OK;
    node_loss_kernel<<<blocks_for(S), 256, 0, (cudaStream_t)stream>>>(per_ray_loss, channels, num_rays, ray_index,
                                                                      node_id, weight, S, num_nodes, loss_sum,
                                                                      weight_sum, dev_error);
    ATDF_LAUNCH_CHECK();
    return ATDF_OK;
}

int atdf_mse_loss(const float* image, const float* target, int64_t count, float scale, double* loss,
                  float* grad_image, float* per_ray_loss, atdf_stream_t stream)
{
    if (count < 0 || (count > 0 && (!image || !target))) return ATDF_ERR_INVALID_ARGUMENT;
    if (loss) ATDF_CUDA_TRY(cudaMemsetAsync(loss, 0, sizeof(double), (cudaStream_t)stream));
    if (count == 0) return ATDF_OK;
    const int64_t nb = div_up(count, 256);
    const unsigned blocks = (unsigned)(nb < 1184 ? nb : 1184);
    mse_kernel<<<blocks, 256, 0, (cudaStream_t)stream>>>(image, target, count, scale, loss, grad_image, per_ray_loss);
    ATDF_LAUNCH_CHECK();
    return ATDF_OK;
}

}  // extern "C"
