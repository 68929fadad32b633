// Fused forward projection and its adjoint in FP32 on the CUDA cores.
//
// A block of 128 threads takes work items (up to kSegItem segments of one
// plane slot) from the item queue and walks each item's samples in tiles of T
// (64 for 64 hidden units, 128 for 32, so that a tile's hidden layer is
// always 4096 values, 8 x 4 per thread). Per tile:
//   geometry   one thread per sample (128 samples at once): t, weight and the
//              coordinates, kept in shared memory;
//   features   one thread per sample and group of 4 channels: 16-byte loads
//              of the texels straight from global memory (L1 / L2);
//   decoder    register-tiled products out of shared memory (simt_gemm.cuh);
//   adjoint    recomputes the tile, keeps the activations' derivatives in
//              registers, holds the weight gradients in registers across all
//              tiles of the block, and adds the factor gradients to global
//              memory with 16-byte vector reductions.
//
// What bounds it: the decoder's FP32 FMAs (5184 a sample forward and 15552 in
// the adjoint for 16 -> 64 -> 64 -> 1). Planes and plane gradients stay out of
// shared memory: on sm_100a a gather of 64-byte texels runs at the same 75-86
// bytes a cycle and SM from L1/L2 as from shared memory, and vector
// reductions into L2 add 4.2 floats a cycle and SM without waiting, where
// shared-memory float atomics (a compare-and-swap loop) add 1.7 to 3.1. That
// leaves room for two blocks an SM in the adjoint of two hidden layers and three
// in the other kernels, whose phases overlap, and lets any block take any item: a slot's items need not share a block.
#pragma once

#include "fused_common.cuh"
#include "simt_gemm.cuh"

namespace atdf {
namespace simt {

constexpr int kThreads = 128;
constexpr int kGeo = 128;  // samples of one geometry pass
constexpr int kMapCap = 2048;  // samples of an item covered by the sample -> segment map (2 KB), where there is room

template <int C, int MODE, int H, int NH>
struct Cfg {
    static constexpr int F = MODE ? 3 * C : C;
    static constexpr int T = 4096 / H;       // samples per tile
    static constexpr int RG = T / 8;         // row groups (8 rows each, interleaved)
    static constexpr int CG = H / 4;         // column groups (4 columns each, interleaved)
    static constexpr int CW = CG / 4;        // warps side by side along the columns
    static constexpr int XP = F + 4;         // pitches
    static constexpr int HP = H + 4;
    static constexpr int V = T * C >= 8 * kThreads ? 2 : 1;  // 4-channel pieces of a texel per thread
    static constexpr int Q = C / (4 * V);    // threads per sample in the gather and scatter
    static constexpr int GI = T * Q / kThreads;  // their samples per thread
    // dW0 [H][F]: 4 x 4 values per thread, the tile's samples split over SG groups of threads
    static constexpr int W0T = H * F / 16;
    static constexpr int SG = 128 / W0T >= 8 ? 8 : 128 / W0T >= 4 ? 4 : 128 / W0T >= 2 ? 2 : 1;
    // dX [T][F]: T / 16 rows x F / 8 columns per thread
    static constexpr int XR = T / 16, XC = F / 8;
    static_assert((H == 64 || H == 32) && C % 8 == 0 && W0T <= 128, "decoder shape");
    static_assert(NH == 1 || (NH == 2 && H == 64), "one or two hidden layers");
};

// Shared-memory layout (float offsets, each a multiple of 4).
template <int C, int MODE, int H, int NH, bool BWD>
struct Smem {
    using K = Cfg<C, MODE, H, NH>;
    static constexpr int w0 = 0;                                      // [H][XP]
    static constexpr int w0t = w0 + H * K::XP;                        // [F][HP]
    static constexpr int w1 = w0t + (BWD ? K::F * K::HP : 0);         // [H][HP]
    static constexpr int w1t = w1 + (NH == 2 ? H * K::HP : 0);        // [H][HP]
    static constexpr int b0 = w1t + (NH == 2 && BWD ? H * K::HP : 0);
    static constexpr int b1 = b0 + H;
    static constexpr int wl = b1 + (NH == 2 ? H : 0);
    static constexpr int bl = wl + H;
    static constexpr int x = bl + 4;                                  // [T][XP]
    static constexpr int h = x + K::T * K::XP;                        // [T][HP]: H0, then dA0
    static constexpr int d = h + (NH == 2 || BWD ? K::T * K::HP : 0);  // [T][HP]: dA1
    static constexpr int geo = d + (NH == 2 && BWD ? K::T * K::HP : 0);  // [6][kGeo], forward also t
    static constexpr int si = geo + (BWD ? 6 : 7) * kGeo;             // [kGeo]
    static constexpr int zrow = BWD ? K::T : kGeo;
    static constexpr int zp = si + kGeo;                              // [CW][zrow]
    static constexpr int dz = zp + K::CW * zrow;                      // [T]
    static constexpr int stash = dz + K::T;                           // adjoint: [GI][3][V][kThreads] float4
    static constexpr int seg = stash + (BWD ? K::GI * 3 * K::V * kThreads * 4 : 0);
    static constexpr int map_cap = BWD && NH == 2 ? 0 : kMapCap;
    static constexpr int total = seg + kSegTabFloats - (kSegMapCap - map_cap) / 4;
    // two blocks an SM (1 KB of each is the system's)
    static_assert(2 * (total * 4 + 1024) <= 228 * 1024 - 1024, "shared memory");
};

// A sample's coordinates in shared memory, and back.
__device__ __forceinline__ void store_geo(float* geo, int s, const SampleGeo& g, float w)
{
    geo[s] = g.lu[0];
    geo[kGeo + s] = g.pu[1];
    geo[2 * kGeo + s] = g.pu[0];
    geo[3 * kGeo + s] = g.pv[0];
    geo[4 * kGeo + s] = g.lu[2];
    geo[5 * kGeo + s] = w;
}

__device__ __forceinline__ SampleGeo load_geo(const float* geo, int s)
{
    const float lx = geo[kGeo + s], ly = geo[2 * kGeo + s], lz = geo[3 * kGeo + s];
    SampleGeo g;
    g.pu[0] = ly;
    g.pv[0] = lz;
    g.pu[1] = lx;
    g.pv[1] = lz;
    g.pu[2] = lx;
    g.pv[2] = ly;
    g.lu[0] = geo[s];
    g.lu[1] = ly;
    g.lu[2] = geo[4 * kGeo + s];
    return g;
}

__device__ __forceinline__ float4 ldg4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }

// Corner offsets (floats) and weights of one sample in plane m and line m.
struct Tap {
    int o[4], l0, l1;
    Corner2 k;
    Corner1 l;
};

template <int C>
__device__ __forceinline__ Tap tap(const FusedParams& p, const SampleGeo& g, int m)
{
    const int Wm = p.field.plane_w[m];
    Tap t;
    t.k = corners2(g.pu[m], g.pv[m], p.field.plane_h[m], Wm);
    t.l = corners1(g.lu[m], p.field.line_len[m]);
    t.o[0] = (t.k.y0 * Wm + t.k.x0) * C;
    t.o[1] = (t.k.y0 * Wm + t.k.x1) * C;
    t.o[2] = (t.k.y1 * Wm + t.k.x0) * C;
    t.o[3] = (t.k.y1 * Wm + t.k.x1) * C;
    t.l0 = t.l.x0 * C;
    t.l1 = t.l.x1 * C;
    return t;
}

// The plane's bilinear values (P: the slot's plane) and the line's linear
// values of the 4 channels at c0.
__device__ __forceinline__ void tap_matrix(const Tap& t, const float* P, int c0, float (&mat)[4])
{
    const float4 nw = ldg4(P + t.o[0] + c0), ne = ldg4(P + t.o[1] + c0), sw = ldg4(P + t.o[2] + c0),
                 se = ldg4(P + t.o[3] + c0);
    mat[0] = bilerp(t.k, nw.x, ne.x, sw.x, se.x);
    mat[1] = bilerp(t.k, nw.y, ne.y, sw.y, se.y);
    mat[2] = bilerp(t.k, nw.z, ne.z, sw.z, se.z);
    mat[3] = bilerp(t.k, nw.w, ne.w, sw.w, se.w);
}

__device__ __forceinline__ void tap_vector(const Tap& t, const float* V, int c0, float (&vec)[4])
{
    const float4 v0 = ldg4(V + t.l0 + c0), v1 = ldg4(V + t.l1 + c0);
    vec[0] = lerp1(t.l, v0.x, v1.x);
    vec[1] = lerp1(t.l, v0.y, v1.y);
    vec[2] = lerp1(t.l, v0.z, v1.z);
    vec[3] = lerp1(t.l, v0.w, v1.w);
}

template <int C>
__device__ __forceinline__ int64_t plane_base(const FusedParams& p, int64_t slot, int m)
{
    return slot * (int64_t)(p.field.plane_h[m] * p.field.plane_w[m] * C);
}

// Features of the tile's samples [s0, s0 + T) of the geometry pass into x
// (zeros for samples past the item's end and outside the region of interest).
// stash (adjoint): the planes' bilinear values, for the line gradients of the
// same thread's samples; gathering them a second time cost as much as the
// features. slots (points): each sample's slot, -1 for zero features.
template <int C, int MODE, int H, int NH, bool STASH>
__device__ __forceinline__ void gather_tile(const FusedParams& p, int64_t slot, bool real, const float* geo, int s0,
                                            int left, float* x, float* stash, const int* slots = nullptr)
{
    using K = Cfg<C, MODE, H, NH>;
    constexpr int V = K::V;
#pragma unroll
    for (int it = 0; it < K::GI; ++it) {
        const int e = threadIdx.x + it * kThreads;
        const int s = e / K::Q, c0 = e % K::Q * 4;  // channels c0 + 4 Q v .. + 3 of piece v
        float f[V][MODE ? 12 : 4];
#pragma unroll
        for (int v = 0; v < V; ++v)
#pragma unroll
            for (int i = 0; i < (MODE ? 12 : 4); ++i) f[v][i] = 0.0f;
        if (slots && s < left) {
            slot = slots[s0 + s];
            real = slot >= 0;
        }
        if (real && s < left) {
            const SampleGeo g = load_geo(geo, s0 + s);
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                const Tap t = tap<C>(p, g, m);
                const float* P = (const float*)p.field.plane[m] + plane_base<C>(p, slot, m);
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    float mat[4], vec[4];
                    tap_matrix(t, P, c0 + 4 * K::Q * v, mat);
                    tap_vector(t, (const float*)p.field.line[m], c0 + 4 * K::Q * v, vec);
                    if (STASH)
                        *reinterpret_cast<float4*>(stash + (((it * 3 + m) * V + v) * kThreads + threadIdx.x) * 4) =
                            make_float4(mat[0], mat[1], mat[2], mat[3]);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float x = __fmul_rn(mat[i], vec[i]);
                        if (MODE)
                            f[v][m * 4 + i] = x;
                        else
                            f[v][i] = m == 0 ? x : __fadd_rn(f[v][i], x);
                    }
                }
            }
        }
#pragma unroll
        for (int v = 0; v < V; ++v)
#pragma unroll
            for (int m = 0; m < (MODE ? 3 : 1); ++m)
                *reinterpret_cast<float4*>(x + s * K::XP + m * C + c0 + 4 * K::Q * v) =
                    make_float4(f[v][m * 4], f[v][m * 4 + 1], f[v][m * 4 + 2], f[v][m * 4 + 3]);
    }
}

template <int C, int MODE, int H, int NH, bool BWD>
__device__ __forceinline__ void load_weights(const FusedParams& p, float* sm)
{
    using K = Cfg<C, MODE, H, NH>;
    using S = Smem<C, MODE, H, NH, BWD>;
    const atdf_mlp_t& m = p.mlp;
    for (int i = threadIdx.x; i < H * K::F; i += kThreads) {
        const int o = i / K::F, k = i % K::F;
        const float v = m.weight[0][i];
        sm[S::w0 + o * K::XP + k] = v;
        if (BWD) sm[S::w0t + k * K::HP + o] = v;
    }
    if (NH == 2)
        for (int i = threadIdx.x; i < H * H; i += kThreads) {
            const int o = i / H, k = i % H;
            const float v = m.weight[1][i];
            sm[S::w1 + o * K::HP + k] = v;
            if (BWD) sm[S::w1t + k * K::HP + o] = v;
        }
    for (int i = threadIdx.x; i < H; i += kThreads) {
        sm[S::b0 + i] = m.bias[0][i];
        if (NH == 2) sm[S::b1 + i] = m.bias[1][i];
        sm[S::wl + i] = m.weight[NH][i];
    }
    if (threadIdx.x == 0) sm[S::bl] = m.bias[NH][0];
}

// The thread's place in the [T][H] tile map: rows rg + i * RG, columns cg + j * CG.
template <class K>
__device__ __forceinline__ void tile_place(int& rg, int& cg, int& cw)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    cw = warp % K::CW;
    rg = lane_row(lane) + 8 * (warp / K::CW);
    cg = lane_col(lane) + 4 * cw;
}

// Geometry of the item's samples [t0, t0 + kGeo), one per thread. dI: keep
// weight * dI (the adjoint's) instead of the weight.
__device__ __forceinline__ void geometry_pass(const FusedParams& p, const SegTab& tab, const ItemInfo& it, int t0,
                                              bool dI, float* geo, int* si)
{
    const int s = threadIdx.x, k = t0 + s;
    if (k < it.total) {
        const SampleState st = sample_state(p, tab, it, k);
        const SampleGeo g = sample_geo_fast(p, &tab, st.node, st.pos);
        store_geo(geo, s, g, dI ? __fmul_rn(tab.acc[st.si], st.w) : st.w);
        si[s] = st.si;
        if (!dI) geo[6 * kGeo + s] = st.t;
    } else {
        geo[5 * kGeo + s] = 0.0f;
        si[s] = -1;
    }
}

// Pre-activations of the first hidden layer for the thread's 8 x 4 values,
// without the bias.
template <int C, int MODE, int H, int NH, bool BWD>
__device__ __forceinline__ void layer0(const float* sm, int rg, int cg, uint64_t (&acc)[8][4])
{
    using K = Cfg<C, MODE, H, NH>;
    using S = Smem<C, MODE, H, NH, BWD>;
    zero2<8, 4>(acc);
    gemm_k<8, 4, K::F>(acc, sm + S::x + rg * K::XP, K::RG * K::XP, sm + S::w0 + cg * K::XP, K::CG * K::XP);
}

// The decoder's hidden layers and the last layer's partial sums (per column
// group, into zp) of the tile whose features are in x.
template <int C, int MODE, int H, int NH>
__device__ __forceinline__ void decode_tile(float* sm, int rg, int cg, int cw, int s0, int hact, float beta)
{
    using K = Cfg<C, MODE, H, NH>;
    using S = Smem<C, MODE, H, NH, false>;
    const int tid = threadIdx.x;
    uint64_t acc[8][4];
    layer0<C, MODE, H, NH, false>(sm, rg, cg, acc);
    // every warp has read all rows of x before any of them gathers the geometry
    // pass's next tile into it (two hidden layers: the barrier after H0)
    if (NH == 1 && K::T < kGeo) __syncthreads();
    if (NH == 2) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float b = sm[S::b0 + cg + j * K::CG];
#pragma unroll
            for (int i = 0; i < 8; ++i)
                sm[S::h + (rg + i * K::RG) * K::HP + cg + j * K::CG] = act_hidden(hact, sum2(acc[i][j]) + b, beta);
        }
        __syncthreads();
        zero2<8, 4>(acc);
        gemm_k<8, 4, H>(acc, sm + S::h + rg * K::HP, K::RG * K::HP, sm + S::w1 + cg * K::HP, K::CG * K::HP);
    }
    // the last layer's sums over the thread's columns
    float z[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int c = cg + j * K::CG;
        const float b = sm[(NH == 2 ? S::b1 : S::b0) + c], wl = sm[S::wl + c];
#pragma unroll
        for (int i = 0; i < 8; ++i) z[i] = fmaf(act_hidden(hact, sum2(acc[i][j]) + b, beta), wl, z[i]);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        z[i] = sum_cols(z[i]);
        if ((tid & 6) == 0) sm[S::zp + cw * S::zrow + s0 + rg + i * K::RG] = z[i];
    }
}

template <int C, int MODE, int H, int NH>
__global__ void __launch_bounds__(kThreads, 3) forward_kernel(FusedParams p)
{
    using K = Cfg<C, MODE, H, NH>;
    using S = Smem<C, MODE, H, NH, false>;
    extern __shared__ __align__(16) float sm[];
    __shared__ int s_ctl[10];
    const int tid = threadIdx.x;
    int rg, cg, cw;
    tile_place<K>(rg, cg, cw);
    if (tid == 0) init_item_queue(s_ctl);
    load_weights<C, MODE, H, NH, false>(p, sm);
    __syncthreads();
    const SegTab tab = seg_tab(sm + S::seg);
    float* geo = sm + S::geo;
    int* si = reinterpret_cast<int*>(sm + S::si);
    const float beta = p.mlp.softplus_beta;
    const int hact = p.mlp.hidden_activation, lact = p.mlp.last_activation;
    while (true) {
        const ItemInfo it = next_item(p, 0, nullptr, tab, nullptr, s_ctl, false, S::map_cap, true);
        if (it.slot < 0) break;
        const bool real = it.slot < p.ws.nslot;
        for (int t0 = 0; t0 < it.total; t0 += kGeo) {
            geometry_pass(p, tab, it, t0, false, geo, si);
            __syncthreads();
            for (int s0 = 0; s0 < kGeo && t0 + s0 < it.total; s0 += K::T) {
                gather_tile<C, MODE, H, NH, false>(p, it.slot, real, geo, s0, it.total - t0 - s0, sm + S::x, nullptr);
                __syncthreads();
                decode_tile<C, MODE, H, NH>(sm, rg, cg, cw, s0, hact, beta);
            }
            __syncthreads();
            {
                float zz = sm[S::bl];
#pragma unroll
                for (int w = 0; w < K::CW; ++w) zz += sm[S::zp + w * S::zrow + tid];
                const int sg = si[tid];
                if (__any_sync(0xffffffffu, sg >= 0)) {
                    const float v = __fmul_rn(act_fwd(lact, zz, beta), geo[5 * kGeo + tid]);
                    // a segment's samples are a run of lanes: its last lane
                    // adds the run's sum to the segment's entry
                    const int lane = tid & 31;
                    float run = sg >= 0 ? v : 0.0f;
#pragma unroll
                    for (int off = 1; off < 32; off <<= 1) {
                        const float o = __shfl_up_sync(0xffffffffu, run, off);
                        const int ko = __shfl_up_sync(0xffffffffu, sg, off);
                        if (lane >= off && ko == sg) run += o;
                    }
                    const int next = __shfl_down_sync(0xffffffffu, sg, 1);
                    if (sg >= 0 && (lane == 31 || next != sg)) atomicAdd(&tab.acc[sg], run);
                    if (sg >= 0 && p.bins) add_to_bins(p, tab, sg, geo[6 * kGeo + tid], v);
                }
            }
            __syncthreads();
        }
        if (tid < it.nseg) p.ws.seg_partial[tab.id[tid]] = tab.acc[tid];
        __syncthreads();
    }
}

// dst[0..3] += w * v[0..3] (16-byte aligned global memory).
__device__ __forceinline__ void red4(float* dst, float w, const float (&v)[4])
{
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(__cvta_generic_to_global(dst)),
                 "f"(__fmul_rn(w, v[0])), "f"(__fmul_rn(w, v[1])), "f"(__fmul_rn(w, v[2])), "f"(__fmul_rn(w, v[3]))
                 : "memory");
}

template <int C, int MODE, int H, int NH>
__global__ void __launch_bounds__(kThreads, NH == 1 ? 3 : 2) backward_kernel(FusedParams p)
{
    using K = Cfg<C, MODE, H, NH>;
    using S = Smem<C, MODE, H, NH, true>;
    constexpr int T = K::T, F = K::F;
    extern __shared__ __align__(16) float sm[];
    __shared__ int s_ctl[10];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int rg, cg, cw;
    tile_place<K>(rg, cg, cw);
    if (tid == 0) init_item_queue(s_ctl);
    load_weights<C, MODE, H, NH, true>(p, sm);
    __syncthreads();
    const SegTab tab = seg_tab(sm + S::seg);
    float* geo = sm + S::geo;
    int* si = reinterpret_cast<int*>(sm + S::si);
    const float beta = p.mlp.softplus_beta;
    const int hact = p.mlp.hidden_activation, lact = p.mlp.last_activation;
    // this block's copy of the line gradients
    const int line_off[3] = {0, p.field.line_len[0] * C, (p.field.line_len[0] + p.field.line_len[1]) * C};
    float* lines = p.ws.seg_partial + (p.line_rep > 0 ? (int)blockIdx.x % p.line_rep : 0) *
                                          (int64_t)(line_off[2] + p.field.line_len[2] * C);

    // decoder gradients held across all tiles: dW1's 8 x 4 and dW0's 4 x 4
    // values of the thread, and its columns' biases and last-layer weights
    uint64_t gw1[4][4], gw0[2][4];
    zero2<4, 4>(gw1);
    zero2<2, 4>(gw0);
    const int o1 = 8 * lane_row(lane), k1 = 4 * (lane_col(lane) + 4 * warp);
    const int u0 = tid % K::W0T, sg0 = tid / K::W0T;
    const int o0 = 4 * (u0 / (F / 4)), c0w = 4 * (u0 % (F / 4));
    float gb0[4] = {0.f, 0.f, 0.f, 0.f}, gb1[4] = {0.f, 0.f, 0.f, 0.f}, gwl[4] = {0.f, 0.f, 0.f, 0.f};
    double gbl = 0.0;  // one scalar summed over every sample: FP64 against cancellation
    const int rx = lane_row(lane) + 8 * (warp & 1), cx = lane_col(lane) + 4 * (warp >> 1);  // dX: rows rx + 16 i, columns cx + 8 j

    while (true) {
        const ItemInfo it = next_item(p, 1, nullptr, tab, nullptr, s_ctl, true, S::map_cap, true);
        if (it.slot < 0) break;
        const bool real = it.slot < p.ws.nslot;
        for (int t0 = 0; t0 < it.total; t0 += kGeo) {
            geometry_pass(p, tab, it, t0, true, geo, si);
            __syncthreads();
            for (int s0 = 0; s0 < kGeo && t0 + s0 < it.total; s0 += T) {
                const int left = it.total - t0 - s0;
                gather_tile<C, MODE, H, NH, true>(p, it.slot, real, geo, s0, left, sm + S::x, sm + S::stash);
                __syncthreads();
                // ---- forward recompute: h and g, the last hidden layer's
                // activation and derivative; g0 the first one's derivative
                float h[8][4], g[8][4], g0[8][4];
                {
                    uint64_t acc[8][4];
                    layer0<C, MODE, H, NH, true>(sm, rg, cg, acc);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float b = sm[S::b0 + cg + j * K::CG];
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            act_pair(hact, sum2(acc[i][j]) + b, beta, h[i][j], g0[i][j]);
                            if (NH == 2) sm[S::h + (rg + i * K::RG) * K::HP + cg + j * K::CG] = h[i][j];
                        }
                    }
                    if (NH == 2) {
                        __syncthreads();
                        zero2<8, 4>(acc);
                        gemm_k<8, 4, H>(acc, sm + S::h + rg * K::HP, K::RG * K::HP, sm + S::w1 + cg * K::HP,
                                        K::CG * K::HP);
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const float b = sm[S::b1 + cg + j * K::CG];
#pragma unroll
                            for (int i = 0; i < 8; ++i)
                                act_pair(hact, sum2(acc[i][j]) + b, beta, h[i][j], g[i][j]);
                        }
                    }
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    float z = 0.0f;
#pragma unroll
                    for (int j = 0; j < 4; ++j) z = fmaf(h[i][j], sm[S::wl + cg + j * K::CG], z);
                    z = sum_cols(z);
                    if ((tid & 6) == 0) sm[S::zp + cw * S::zrow + rg + i * K::RG] = z;
                }
                __syncthreads();
                if (tid < T) {
                    float z = sm[S::bl];
#pragma unroll
                    for (int w = 0; w < K::CW; ++w) z += sm[S::zp + w * S::zrow + tid];
                    const float dz = geo[5 * kGeo + s0 + tid] * act_grad(lact, z, beta);
                    sm[S::dz + tid] = dz;
                    gbl += (double)dz;
                }
                __syncthreads();
                // ---- last layer's gradients, dA of the last hidden layer
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int c = cg + j * K::CG;
                    const float wl = sm[S::wl + c];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int row = rg + i * K::RG;
                        const float dz = sm[S::dz + row];
                        gwl[j] = fmaf(dz, h[i][j], gwl[j]);
                        const float da = dz * wl * (NH == 2 ? g[i][j] : g0[i][j]);
                        (NH == 2 ? gb1[j] : gb0[j]) += da;
                        sm[(NH == 2 ? S::d : S::h) + row * K::HP + c] = da;
                    }
                }
                __syncthreads();
                if (NH == 2) {
                    gemm_s<4, 4>(gw1, sm + S::d + o1, K::HP, sm + S::h + k1, K::HP, T);
                    uint64_t acc[8][4];
                    zero2<8, 4>(acc);
                    gemm_k<8, 4, H>(acc, sm + S::d + rg * K::HP, K::RG * K::HP, sm + S::w1t + cg * K::HP,
                                    K::CG * K::HP);
                    __syncthreads();
#pragma unroll
                    for (int j = 0; j < 4; ++j)
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const float da = sum2(acc[i][j]) * g0[i][j];
                            gb0[j] += da;
                            sm[S::h + (rg + i * K::RG) * K::HP + cg + j * K::CG] = da;
                        }
                    __syncthreads();
                }
                // ---- dW0 and dX from dA0
                if (sg0 < K::SG)
                    gemm_s<2, 4>(gw0, sm + S::h + sg0 * (T / K::SG) * K::HP + o0, K::HP,
                                 sm + S::x + sg0 * (T / K::SG) * K::XP + c0w, K::XP, T / K::SG);
                {
                    uint64_t acc[K::XR][K::XC];
                    zero2<K::XR, K::XC>(acc);
                    gemm_k<K::XR, K::XC, H>(acc, sm + S::h + rx * K::HP, 16 * K::HP, sm + S::w0t + cx * K::HP,
                                            8 * K::HP);
                    __syncthreads();
#pragma unroll
                    for (int i = 0; i < K::XR; ++i)
#pragma unroll
                        for (int j = 0; j < K::XC; ++j)
                            sm[S::x + (rx + 16 * i) * K::XP + cx + 8 * j] = sum2(acc[i][j]);
                }
                __syncthreads();
                // ---- factor gradients; the next tile's features go into the
                // entries of x that the same thread reads here
                if (!real) continue;
#pragma unroll
                for (int e0 = 0; e0 < K::GI; ++e0) {
                    const int e = tid + e0 * kThreads;
                    const int s = e / K::Q, c0 = e % K::Q * 4;
                    if (s >= left) continue;
                    const SampleGeo ge = load_geo(geo, s0 + s);
#pragma unroll
                    for (int m = 0; m < 3; ++m) {
                        const Tap t = tap<C>(p, ge, m);
                        const int64_t base = plane_base<C>(p, it.slot, m);
                        float* GP = p.gfield.plane[m] + base;
#pragma unroll
                        for (int v = 0; v < K::V; ++v) {
                            const int c = c0 + 4 * K::Q * v;
                            float vec[4];
                            tap_vector(t, (const float*)p.field.line[m], c, vec);
                            const float4 mat = *reinterpret_cast<const float4*>(
                                sm + S::stash + (((e0 * 3 + m) * K::V + v) * kThreads + tid) * 4);
                            const float4 gf = *reinterpret_cast<const float4*>(sm + S::x + s * K::XP + (MODE ? m * C : 0) + c);
                            const float gm[4] = {__fmul_rn(gf.x, vec[0]), __fmul_rn(gf.y, vec[1]),
                                                 __fmul_rn(gf.z, vec[2]), __fmul_rn(gf.w, vec[3])};
                            const float gv[4] = {__fmul_rn(gf.x, mat.x), __fmul_rn(gf.y, mat.y),
                                                 __fmul_rn(gf.z, mat.z), __fmul_rn(gf.w, mat.w)};
                            red4(GP + t.o[0] + c, t.k.w_nw, gm);
                            red4(GP + t.o[1] + c, t.k.w_ne, gm);
                            red4(GP + t.o[2] + c, t.k.w_sw, gm);
                            red4(GP + t.o[3] + c, t.k.w_se, gm);
                            if (p.line_rep > 0) {
                                red4(lines + line_off[m] + t.l0 + c, t.l.w0, gv);
                                red4(lines + line_off[m] + t.l1 + c, t.l.w1, gv);
                            } else {
#pragma unroll
                                for (int i = 0; i < 4; ++i) {
                                    atomicAdd(p.gfield.line[m] + t.l0 + c + i, __fmul_rn(t.l.w0, gv[i]));
                                    atomicAdd(p.gfield.line[m] + t.l1 + c + i, __fmul_rn(t.l.w1, gv[i]));
                                }
                            }
                        }
                    }
                }
            }
            __syncthreads();
        }
    }

    // flush the decoder gradients
    if (NH == 2)
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float lo, hi;
                unpack2(gw1[i][j], lo, hi);
                atomicAdd(&p.gmlp.weight[1][(o1 + 2 * i) * H + k1 + j], lo);
                atomicAdd(&p.gmlp.weight[1][(o1 + 2 * i + 1) * H + k1 + j], hi);
            }
    // dW0's sample groups first add up in shared memory (x is free now): one
    // global atomic per weight and block, since all blocks meet on the same
    // few addresses here
    for (int gg = 0; gg < K::SG; ++gg) {
        if (sg0 == gg)
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    float lo, hi;
                    unpack2(gw0[i][j], lo, hi);
                    float* q = sm + S::x + (o0 + 2 * i) * F + c0w + j;
                    q[0] = gg == 0 ? lo : q[0] + lo;
                    q[F] = gg == 0 ? hi : q[F] + hi;
                }
        __syncthreads();
    }
    for (int i = tid; i < H * F; i += kThreads) atomicAdd(&p.gmlp.weight[0][i], sm[S::x + i]);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        gwl[j] = sum_rows(gwl[j]);
        gb0[j] = sum_rows(gb0[j]);
        gb1[j] = sum_rows(gb1[j]);
    }
    if (lane_row(lane) == 0)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int c = cg + j * K::CG;
            atomicAdd(&p.gmlp.weight[NH][c], gwl[j]);
            atomicAdd(&p.gmlp.bias[0][c], gb0[j]);
            if (NH == 2) atomicAdd(&p.gmlp.bias[1][c], gb1[j]);
        }
    for (int off = 16; off > 0; off >>= 1) gbl += __shfl_down_sync(0xffffffffu, gbl, off);
    if (lane == 0) atomicAdd(p.ws.last_sum, gbl);
}

// Density at points with known leaves (field and decoder in one pass, no
// gradients): the forward's tiles with the geometry of points instead of the
// samples of segments. Bound by the decoder like the forward.
struct PointArgs {
    const float* pos;     // [S, 3]
    const int64_t* node;  // [S]
    int64_t S;
    float* out;  // [S]
};

template <int C, int MODE, int H, int NH>
__global__ void __launch_bounds__(kThreads, 3) points_kernel(FusedParams p, PointArgs a)
{
    using K = Cfg<C, MODE, H, NH>;
    using S = Smem<C, MODE, H, NH, false>;
    extern __shared__ __align__(16) float sm[];
    const int tid = threadIdx.x;
    int rg, cg, cw;
    tile_place<K>(rg, cg, cw);
    load_weights<C, MODE, H, NH, false>(p, sm);
    float* geo = sm + S::geo;
    int* slots = reinterpret_cast<int*>(sm + S::si);
    const float beta = p.mlp.softplus_beta;
    const int hact = p.mlp.hidden_activation, lact = p.mlp.last_activation;
    for (int64_t t0 = (int64_t)blockIdx.x * kGeo; t0 < a.S; t0 += (int64_t)gridDim.x * kGeo) {
        const int left = (int)min((int64_t)kGeo, a.S - t0);
        __syncthreads();
        int slot = -1;
        if (tid < left) {
            const int64_t i = t0 + tid, nd = a.node[i];
            if (nd < 0 || nd >= p.tree.num_nodes) {
                set_err(p.err, ATDF_DEVERR_INDEX);
            } else {
                const int64_t s = p.field.leaf_slot[nd];
                if (s >= p.field.num_slots) set_err(p.err, ATDF_DEVERR_INDEX);
                if (s >= 0 && s < p.field.num_slots) {
                    slot = (int)s;
                    const float pos[3] = {a.pos[3 * i], a.pos[3 * i + 1], a.pos[3 * i + 2]};
                    store_geo(geo, tid, sample_geo(pos, p.tree.node_position_min + 3 * nd,
                                                   p.tree.node_position_max + 3 * nd, p.field.roi_min,
                                                   p.field.roi_max), 0.0f);
                }
            }
        }
        slots[tid] = slot;
        __syncthreads();
        for (int s0 = 0; s0 < left; s0 += K::T) {
            gather_tile<C, MODE, H, NH, false>(p, 0, false, geo, s0, left - s0, sm + S::x, nullptr, slots);
            __syncthreads();
            decode_tile<C, MODE, H, NH>(sm, rg, cg, cw, s0, hact, beta);
        }
        __syncthreads();
        if (tid < left) {
            float z = sm[S::bl];
#pragma unroll
            for (int w = 0; w < K::CW; ++w) z += sm[S::zp + w * S::zrow + tid];
            a.out[t0 + tid] = act_fwd(lact, z, beta);
        }
    }
}

}  // namespace simt
}  // namespace atdf
