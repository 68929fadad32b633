// The decoder MLP as an operator on its own (DecodeFeatures): FP32 on the CUDA
// cores for any layer widths up to 256.
//
// Reference: hyperacorn/csrc/geometry/Modules.h:23-149, geometry.cpp:176-253.
//
// A block of NT threads keeps every layer's weights in shared memory and walks
// tiles of T = NT / 16 * RM rows (RM rows x 4 columns of outputs a thread,
// simt_gemm.cuh). The adjoint recomputes a tile's layers, keeping each
// layer's activation and derivative in shared memory, and sums the weight
// gradients there over all tiles of the block: one global atomic per weight
// and block instead of one per weight and row. Both are bound by the FP32
// FMAs and the shared loads that feed them. Networks whose tile does not fit
// in shared memory (several 256-wide layers) take the one-thread-a-row
// kernels.

#include <algorithm>
#include <cfloat>
#include <type_traits>

#include "atdf_common.cuh"
#include "simt_gemm.cuh"

namespace atdf {
namespace mlp {

constexpr int kMaxWidth = 256;
constexpr int kMaxPre = 1024;  // hidden and output values of one row in the one-thread-a-row adjoint

__host__ __device__ constexpr int round4(int n) { return (n + 3) & ~3; }
// Row pitch of a matrix with n columns: a multiple of 4, and 4 mod 8, so that
// the 16-byte loads of rows side by side fall into distinct banks.
__host__ __device__ constexpr int pitch_of(int n) { return round4(n) % 8 == 4 ? round4(n) : round4(n) + 4; }
// Columns that the tile products write for n outputs: blocks of 64, then one
// of 32 or 16; up to 4 outputs are plain dot products.
__host__ __device__ constexpr int cols_of(int n)
{
    if (n <= 4) return 4;
    const int full = n / 64 * 64, rest = n - full;
    return full + (rest == 0 ? 0 : rest <= 16 ? 16 : rest <= 32 ? 32 : 64);
}

// Shared-memory layout (float offsets) of a network.
struct Plan {
    int w[ATDF_MAX_LAYERS];   // weights [cols_of(out)][pitch_of(in)], zero padded
    int b[ATDF_MAX_LAYERS];   // biases [cols_of(out)]
    int wt[ATDF_MAX_LAYERS];  // adjoint: transposed weights [cols_of(in)][pitch_of(out)]
    int gw[ATDF_MAX_LAYERS];  // adjoint: weight gradients [round8(out)][pitch_of(in)]
    int gb[ATDF_MAX_LAYERS];  // adjoint: bias gradients [round4(out)]
    int h[ATDF_MAX_LAYERS];   // inputs of layer l [T][pitch_of(in)]
    int d[ATDF_MAX_LAYERS];   // adjoint: derivative, then dA of layer l [T][pitch_of(out)]
    int total;
};

static Plan make_plan(const atdf_mlp_t& m, int T, bool bwd)
{
    Plan p;
    int o = 0;
    auto take = [&](int n) {
        const int at = o;
        o += round4(n);
        return at;
    };
    for (int l = 0; l < m.num_layers; ++l) {
        const int in = m.dims[l], on = m.dims[l + 1];
        p.w[l] = take(cols_of(on) * pitch_of(in));
        p.b[l] = take(cols_of(on));
        p.wt[l] = bwd ? take(cols_of(in) * pitch_of(on)) : 0;
        p.gw[l] = bwd ? take(((on + 7) & ~7) * pitch_of(in)) : 0;
        p.gb[l] = bwd ? take(on) : 0;
    }
    if (bwd) {
        for (int l = 0; l < m.num_layers; ++l) {
            p.h[l] = take(T * pitch_of(m.dims[l]));
            p.d[l] = take(T * pitch_of(m.dims[l + 1]) + 4);  // weight_gradient reads 8 columns at a time
        }
    } else {  // two buffers in turn
        int widest = 0;
        for (int l = 0; l < m.num_layers; ++l) widest = std::max(widest, pitch_of(m.dims[l]));
        const int a = take(T * widest), b = m.num_layers > 1 ? take(T * widest) : a;
        for (int l = 0; l < m.num_layers; ++l) p.h[l] = l & 1 ? b : a;
    }
    p.total = o;
    return p;
}

template <int NT>
__device__ void load_weights(const atdf_mlp_t& m, const Plan& pl, float* sm, bool bwd)
{
    for (int l = 0; l < m.num_layers; ++l) {
        const int in = m.dims[l], on = m.dims[l + 1], ip = pitch_of(in), op = pitch_of(on);
        const float* W = m.weight[l];
        for (int i = threadIdx.x; i < cols_of(on) * ip; i += NT) {
            const int o = i / ip, k = i % ip;
            sm[pl.w[l] + i] = o < on && k < in ? W[o * in + k] : 0.0f;
        }
        for (int i = threadIdx.x; i < cols_of(on); i += NT) sm[pl.b[l] + i] = i < on ? m.bias[l][i] : 0.0f;
        if (!bwd) continue;
        for (int i = threadIdx.x; i < cols_of(in) * op; i += NT) {
            const int k = i / op, o = i % op;
            sm[pl.wt[l] + i] = o < on && k < in ? W[o * in + k] : 0.0f;
        }
        for (int i = threadIdx.x; i < ((on + 7) & ~7) * ip; i += NT) sm[pl.gw[l] + i] = 0.0f;
        for (int i = threadIdx.x; i < round4(on); i += NT) sm[pl.gb[l] + i] = 0.0f;
    }
}

// Rows [row0, row0 + T) of x [S][n] into dst [T][pitch] (zeros past S and in
// the columns n .. round4(n)).
template <int NT, int T>
__device__ __forceinline__ void load_rows(const float* __restrict__ x, int64_t row0, int64_t S, int n, float* dst)
{
    const int pitch = pitch_of(n), n4 = round4(n) / 4;
    const bool vec = n % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
    for (int i = threadIdx.x; i < T * n4; i += NT) {
        const int r = i / n4, c = i % n4 * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row0 + r < S) {
            const float* src = x + (row0 + r) * n + c;
            if (vec) {
                v = __ldg(reinterpret_cast<const float4*>(src));
            } else {
                v.x = src[0];
                if (c + 1 < n) v.y = src[1];
                if (c + 2 < n) v.z = src[2];
                if (c + 3 < n) v.w = src[3];
            }
        }
        *reinterpret_cast<float4*>(dst + r * pitch + c) = v;
    }
}

// acc = A B^T for RM rows (row0 + RG i) and CN columns (col0 + 16 j), K contiguous.
template <int RG, int RM, int CN>
__device__ __forceinline__ void tile_product(uint64_t (&acc)[RM][CN], const float* a, int ap, const float* b, int bp,
                                             int K)
{
    zero2<RM, CN>(acc);
#pragma unroll 2
    for (int k = 0; k < K; k += 4) {
        ulonglong2 av[RM], bv[CN];
#pragma unroll
        for (int i = 0; i < RM; ++i) av[i] = *reinterpret_cast<const ulonglong2*>(a + i * RG * ap + k);
#pragma unroll
        for (int j = 0; j < CN; ++j) bv[j] = *reinterpret_cast<const ulonglong2*>(b + j * 16 * bp + k);
#pragma unroll
        for (int i = 0; i < RM; ++i)
#pragma unroll
            for (int j = 0; j < CN; ++j) {
                acc[i][j] = ffma2(av[i].x, bv[j].x, acc[i][j]);
                acc[i][j] = ffma2(av[i].y, bv[j].y, acc[i][j]);
            }
    }
}

// One layer's tile: out(row, column, value, real) for every value A B^T (+ bias
// per column) of the T rows and the columns up to round4(n), the ones past n
// with real false; A [T][ap], B [cols_of(n)][bp], contraction over K (a
// multiple of 4, zero padded).
template <int NT, int RM, class Out>
__device__ __forceinline__ void tile_layer(const float* A, int ap, const float* B, int bp, int K, int n,
                                           const float* bias, Out out)
{
    constexpr int RG = NT / 16, T = RG * RM;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (n <= 4) {  // dot products: one row and output at a time
        for (int e = threadIdx.x; e < T * 4; e += NT) {
            const int r = e % T, c = e / T;
            float s = 0.0f;
            if (c < n)
                for (int k = 0; k < K; k += 4) {
                    const float4 a = *reinterpret_cast<const float4*>(A + r * ap + k);
                    const float4 b = *reinterpret_cast<const float4*>(B + c * bp + k);
                    s = fmaf(a.x, b.x, s);
                    s = fmaf(a.y, b.y, s);
                    s = fmaf(a.z, b.z, s);
                    s = fmaf(a.w, b.w, s);
                }
            out(r, c, bias ? s + bias[c] : s, c < n);
        }
        return;
    }
    const int rg = lane_row(lane) + 8 * (warp >> 2), cg = lane_col(lane) + 4 * (warp & 3);
    const float* a = A + rg * ap;
    for (int c0 = 0; c0 < n; c0 += 64) {
        const float* b = B + (c0 + cg) * bp;
        auto write = [&](auto& acc, auto cn) {
#pragma unroll
            for (int j = 0; j < decltype(cn)::value; ++j) {
                const int c = c0 + cg + 16 * j;
                if (c >= round4(n)) continue;
                const float bj = bias ? bias[c] : 0.0f;
                if (c < n) {
#pragma unroll
                    for (int i = 0; i < RM; ++i) out(rg + RG * i, c, sum2(acc[i][j]) + bj, true);
                } else {
#pragma unroll
                    for (int i = 0; i < RM; ++i) out(rg + RG * i, c, 0.0f, false);
                }
            }
        };
        if (n - c0 > 32) {
            uint64_t acc[RM][4];
            tile_product<RG, RM, 4>(acc, a, ap, b, bp, K);
            write(acc, std::integral_constant<int, 4>());
        } else if (n - c0 > 16) {
            uint64_t acc[RM][2];
            tile_product<RG, RM, 2>(acc, a, ap, b, bp, K);
            write(acc, std::integral_constant<int, 2>());
        } else {
            uint64_t acc[RM][1];
            tile_product<RG, RM, 1>(acc, a, ap, b, bp, K);
            write(acc, std::integral_constant<int, 1>());
        }
    }
}

template <int NT, int RM>
__global__ void __launch_bounds__(NT, 384 / NT)
    forward_kernel(atdf_mlp_t m, Plan pl, const float* __restrict__ x, int64_t S, float* __restrict__ out)
{
    constexpr int T = NT / 16 * RM;
    extern __shared__ __align__(16) float sm[];
    load_weights<NT>(m, pl, sm, false);
    const int L = m.num_layers, last_n = m.dims[L];
    for (int64_t row0 = (int64_t)blockIdx.x * T; row0 < S; row0 += (int64_t)gridDim.x * T) {
        __syncthreads();
        load_rows<NT, T>(x, row0, S, m.dims[0], sm + pl.h[0]);
        __syncthreads();
        for (int l = 0; l < L; ++l) {
            const int in = m.dims[l], on = m.dims[l + 1], np = pitch_of(on);
            const float* bias = sm + pl.b[l];
            if (l == L - 1) {
                tile_layer<NT, RM>(sm + pl.h[l], pitch_of(in), sm + pl.w[l], pitch_of(in), round4(in), on, bias,
                                   [&](int r, int c, float v, bool real) {
                                       if (real && row0 + r < S)
                                           out[(row0 + r) * last_n + c] =
                                               act_hidden(m.last_activation, v, m.softplus_beta);
                                   });
            } else {
                float* h = sm + pl.h[l + 1];
                tile_layer<NT, RM>(sm + pl.h[l], pitch_of(in), sm + pl.w[l], pitch_of(in), round4(in), on, bias,
                                   [&](int r, int c, float v, bool real) {
                                       h[r * np + c] = real ? act_hidden(m.hidden_activation, v, m.softplus_beta) : 0.0f;
                                   });
                __syncthreads();
            }
        }
    }
}

// gW [on][ip] += D^T H over the tile's T rows: 8 x 4 values a thread; where
// that leaves threads idle, the rows are split over groups of threads, which
// add their sums one after the other. skip_zeros: without the products of a
// zero in D, a thread a weight as for few outputs.
template <int NT, int T>
__device__ __forceinline__ void weight_gradient(const float* D, int dp, const float* H, int ip, int in, int on,
                                                float* gw, bool skip_zeros)
{
    if (on <= 4 || skip_zeros) {  // a thread per weight (and group of rows)
        const int n = on * in, g = max(1, min(NT / n, T / 8)), per = (T + g - 1) / g;
        for (int e = threadIdx.x; e < n * g; e += NT) {
            const int o = e % n / in, k = e % n % in, s0 = e / n * per, s1 = min(T, s0 + per);
            float s = 0.0f;
            if (skip_zeros) {
                for (int r = s0; r < s1; ++r) {
                    const float d = D[r * dp + o];
                    if (d != 0.0f) s = fmaf(d, H[r * ip + k], s);
                }
            } else {
                for (int r = s0; r < s1; ++r) s = fmaf(D[r * dp + o], H[r * ip + k], s);
            }
            atomicAdd(&gw[o * ip + k], s);
        }
        __syncthreads();
        return;
    }
    const int kb = (in + 3) / 4, tiles = (on + 7) / 8 * kb;
    const int groups = tiles <= NT / 4 ? 4 : tiles <= NT / 2 ? 2 : 1, rows = T / groups;
    for (int u0 = 0; u0 < tiles * groups; u0 += NT) {
        const int u = u0 + threadIdx.x, t = u % tiles, g = u / tiles;
        const int o = t / kb * 8, k = t % kb * 4;
        uint64_t acc[4][4];
        zero2<4, 4>(acc);
        if (g < groups) gemm_s<4, 4>(acc, D + g * rows * dp + o, dp, H + g * rows * ip + k, ip, rows);
        for (int gg = 0; gg < groups; ++gg) {
            if (g == gg) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    float lo[4], hi[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) unpack2(acc[i][j], lo[j], hi[j]);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        float4* q = reinterpret_cast<float4*>(gw + (o + 2 * i + h) * ip + k);
                        const float* v = h ? hi : lo;
                        float4 w = *q;
                        w.x += v[0];
                        w.y += v[1];
                        w.z += v[2];
                        w.w += v[3];
                        *q = w;
                    }
                }
            }
            __syncthreads();
        }
    }
}

template <int NT, int RM>
__global__ void __launch_bounds__(NT, NT == 128 ? 3 : 1)
    backward_kernel(atdf_mlp_t m, Plan pl, const float* __restrict__ x, int64_t S, const float* __restrict__ gout,
                    float* __restrict__ gx, atdf_mlp_grad_t gr)
{
    constexpr int T = NT / 16 * RM;
    extern __shared__ __align__(16) float sm[];
    load_weights<NT>(m, pl, sm, true);
    const int L = m.num_layers, last_n = m.dims[L];
    // The products of a row that wants no gradient count as nothing, also with
    // infinite or NaN inputs. The fast products add 0 * input like any other, so
    // a block whose sums are not finite takes its rows again without the zeros.
    for (bool skip_zeros = false;; skip_zeros = true) {
        for (int64_t row0 = (int64_t)blockIdx.x * T; row0 < S; row0 += (int64_t)gridDim.x * T) {
            __syncthreads();
            load_rows<NT, T>(x, row0, S, m.dims[0], sm + pl.h[0]);
            __syncthreads();
            // forward: h[l + 1] = activation, d[l] = derivative (last layer: dA)
            for (int l = 0; l < L; ++l) {
                const int in = m.dims[l], on = m.dims[l + 1], np = pitch_of(on);
                const bool last = l == L - 1;
                const float* bias = sm + pl.b[l];
                float* d = sm + pl.d[l];
                float* h = sm + (last ? 0 : pl.h[l + 1]);
                const int act = last ? m.last_activation : m.hidden_activation;
                tile_layer<NT, RM>(sm + pl.h[l], pitch_of(in), sm + pl.w[l], pitch_of(in), round4(in), on, bias,
                                   [&](int r, int c, float v, bool real) {
                                       float act_v = 0.0f, g = 0.0f;
                                       if (real) act_pair(act, v, m.softplus_beta, act_v, g);
                                       if (last)
                                           g = real && row0 + r < S ? g * gout[(row0 + r) * last_n + c] : 0.0f;
                                       else
                                           h[r * np + c] = act_v;
                                       d[r * np + c] = g;
                                   });
                __syncthreads();
            }
            // adjoint, last layer first: d[l] holds dA
            for (int l = L - 1; l >= 0; --l) {
                const int in = m.dims[l], on = m.dims[l + 1], ip = pitch_of(in), op = pitch_of(on);
                const float* D = sm + pl.d[l];
                {  // bias: column sums, a thread per output and group of rows
                    const int g = max(1, min(NT / on, T / 8)), per = (T + g - 1) / g;
                    for (int e = threadIdx.x; e < on * g; e += NT) {
                        const int o = e % on, s0 = e / on * per, s1 = min(T, s0 + per);
                        float s = 0.0f;
                        for (int r = s0; r < s1; ++r) s += D[r * op + o];
                        atomicAdd(&sm[pl.gb[l] + o], s);
                    }
                }
                if (l > 0 || gx) {
                    float* dn = sm + (l > 0 ? pl.d[l - 1] : 0);
                    tile_layer<NT, RM>(D, op, sm + pl.wt[l], op, round4(on), in, nullptr, [&](int r, int c, float v, bool real) {
                        if (!real) return;
                        if (l > 0) {  // the derivative there is read and replaced by this thread alone
                            dn[r * ip + c] *= v;
                        } else if (row0 + r < S) {
                            gx[(row0 + r) * in + c] = v;
                        }
                    });
                }
                weight_gradient<NT, T>(D, op, sm + pl.h[l], ip, in, on, sm + pl.gw[l], skip_zeros);
            }
        }
        __syncthreads();
        float wild = 0.0f;  // NaN as soon as a sum (or a padding column's product) is not finite
        for (int l = 0; l < L; ++l)
            for (int i = threadIdx.x * 4; i < m.dims[l + 1] * pitch_of(m.dims[l]); i += NT * 4) {
                const float4 v = *reinterpret_cast<const float4*>(sm + pl.gw[l] + i);
                wild += v.x * 0.0f + v.y * 0.0f + v.z * 0.0f + v.w * 0.0f;
            }
        if (__syncthreads_and(wild == 0.0f) || skip_zeros) break;
        for (int l = 0; l < L; ++l) {
            const int on = m.dims[l + 1];
            for (int i = threadIdx.x; i < ((on + 7) & ~7) * pitch_of(m.dims[l]); i += NT) sm[pl.gw[l] + i] = 0.0f;
            for (int i = threadIdx.x; i < on; i += NT) sm[pl.gb[l] + i] = 0.0f;
        }
    }
    for (int l = 0; l < L; ++l) {
        const int in = m.dims[l], on = m.dims[l + 1], ip = pitch_of(in);
        if (gr.weight[l])
            for (int i = threadIdx.x; i < on * in; i += NT)
                atomicAdd(&gr.weight[l][i], sm[pl.gw[l] + i / in * ip + i % in]);
        if (gr.bias[l])
            for (int i = threadIdx.x; i < on; i += NT) atomicAdd(&gr.bias[l][i], sm[pl.gb[l] + i]);
    }
}

// One thread per row, for networks too wide for the tile kernels.
__global__ void row_forward_kernel(atdf_mlp_t m, const float* __restrict__ x, int64_t S, float* __restrict__ out)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= S) return;
    float buf[2][kMaxWidth];
    const int in0 = m.dims[0];
    for (int k = 0; k < in0; ++k) buf[0][k] = x[i * in0 + k];
    int cur = 0;
    for (int l = 0; l < m.num_layers; ++l) {
        const int in = m.dims[l], on = m.dims[l + 1];
        const bool last = l == m.num_layers - 1;
        const float* Wl = m.weight[l];
        for (int o = 0; o < on; ++o) {
            float acc = 0.0f;
            for (int k = 0; k < in; ++k) acc = fmaf(buf[cur][k], Wl[o * in + k], acc);
            acc += m.bias[l][o];
            buf[cur ^ 1][o] = act_fwd(last ? m.last_activation : m.hidden_activation, acc, m.softplus_beta);
        }
        cur ^= 1;
    }
    const int on = m.dims[m.num_layers];
    for (int o = 0; o < on; ++o) out[i * on + o] = buf[cur][o];
}

__global__ void row_backward_kernel(atdf_mlp_t m, const float* __restrict__ x, int64_t S, const float* __restrict__ gout,
                               float* __restrict__ gx, atdf_mlp_grad_t gr)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= S) return;
    float pre[kMaxPre];
    float g[2][kMaxWidth];
    int po[ATDF_MAX_LAYERS + 1];
    po[0] = 0;
    for (int l = 0; l < m.num_layers; ++l) po[l + 1] = po[l] + m.dims[l + 1];
    const int in0 = m.dims[0];
    // forward keeping pre-activations
    for (int l = 0; l < m.num_layers; ++l) {
        const int in = m.dims[l], on = m.dims[l + 1];
        const float* Wl = m.weight[l];
        for (int o = 0; o < on; ++o) {
            float acc = 0.0f;
            for (int k = 0; k < in; ++k) {
                const float xin = l == 0 ? x[i * in0 + k]
                                         : act_fwd(m.hidden_activation, pre[po[l - 1] + k], m.softplus_beta);
                acc = fmaf(xin, Wl[o * in + k], acc);
            }
            pre[po[l] + o] = acc + m.bias[l][o];
        }
    }
    const int L = m.num_layers;
    int cur = 0;
    for (int o = 0; o < m.dims[L]; ++o) g[cur][o] = gout[i * m.dims[L] + o];
    for (int l = L - 1; l >= 0; --l) {
        const int in = m.dims[l], on = m.dims[l + 1];
        const int a = l == L - 1 ? m.last_activation : m.hidden_activation;
        for (int o = 0; o < on; ++o) g[cur][o] *= act_grad(a, pre[po[l] + o], m.softplus_beta);
        const float* Wl = m.weight[l];
        for (int o = 0; o < on; ++o) {
            const float gp = g[cur][o];
            if (gr.bias[l]) atomicAdd(&gr.bias[l][o], gp);
            if (gr.weight[l] && gp != 0.0f) {
                for (int k = 0; k < in; ++k) {
                    const float xin = l == 0 ? x[i * in0 + k]
                                             : act_fwd(m.hidden_activation, pre[po[l - 1] + k], m.softplus_beta);
                    atomicAdd(&gr.weight[l][o * in + k], gp * xin);
                }
            }
        }
        for (int k = 0; k < in; ++k) {
            float acc = 0.0f;
            for (int o = 0; o < on; ++o) acc = fmaf(g[cur][o], Wl[o * in + k], acc);
            g[cur ^ 1][k] = acc;
        }
        cur ^= 1;
    }
    if (gx)
        for (int k = 0; k < in0; ++k) gx[i * in0 + k] = g[cur][k];
}

}  // namespace mlp
}  // namespace atdf

using namespace atdf;

static bool mlp_ok(const atdf_mlp_t* m)
{
    if (!m || m->num_layers <= 0 || m->num_layers > ATDF_MAX_LAYERS) return false;
    int total = 0;
    for (int l = 0; l <= m->num_layers; ++l) {
        if (m->dims[l] <= 0 || m->dims[l] > mlp::kMaxWidth) return false;
        if (l > 0) total += m->dims[l];
    }
    for (int l = 0; l < m->num_layers; ++l)
        if (!m->weight[l] || !m->bias[l]) return false;
    return total <= mlp::kMaxPre;
}

// The kernel variants (threads and rows a thread) in order of preference.
// Blocks of 128 threads come first: several share an SM, so that one's phases
// (loads, products, gradients) overlap another's; the taller the tile, the
// fewer shared loads per FMA. 256 threads share one copy of the weights where
// two blocks of 128 would not fit.
struct Shape {
    int nt, rm;
};
static const Shape kForward[] = {{128, 8}, {128, 4}, {128, 2}};
static const Shape kBackward[] = {{128, 8}, {128, 4}, {256, 8}, {256, 4}, {256, 2}};

// The first variant that fits in shared memory, gives every SM a tile and, for
// 128 threads, puts two blocks on an SM; else the last one that fits (-1: none).
template <int N>
static int pick_shape(const Shape (&shapes)[N], const atdf_mlp_t& m, int64_t S, bool bwd, int sms, int optin,
                      mlp::Plan& plan)
{
    int found = -1;
    for (int i = 0; i < N; ++i) {
        const int T = shapes[i].nt / 16 * shapes[i].rm;
        const mlp::Plan p = mlp::make_plan(m, T, bwd);
        if (p.total * 4 > optin) continue;
        if (bwd && shapes[i].nt == 128 && 2 * (p.total * 4 + 1024) > optin) continue;
        found = i;
        plan = p;
        if (div_up(S, T) >= sms) break;
    }
    return found;
}

template <class Fn, class... Args>
static int launch_tiles(Fn fn, Shape sh, const mlp::Plan& plan, int64_t S, int sms, cudaStream_t st, Args... args)
{
    const int smem = plan.total * 4;
    if (const int e = allow_dynamic_shared((const void*)fn, smem)) return e;
    int per = 0;
    ATDF_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, (const void*)fn, sh.nt, smem));
    if (per < 1) return ATDF_ERR_CUDA;
    fn<<<(unsigned)std::min<int64_t>(div_up(S, sh.nt / 16 * sh.rm), (int64_t)sms * per), sh.nt, smem, st>>>(args...);
    ATDF_LAUNCH_CHECK();
    return ATDF_OK;
}

static int device_limits(int& sms, int& optin)
{
    int dev = 0;
    ATDF_CUDA_TRY(cudaGetDevice(&dev));
    ATDF_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    ATDF_CUDA_TRY(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    return ATDF_OK;
}

extern "C" {

int atdf_mlp_forward(const atdf_mlp_t* mlp, const float* x, int64_t S, float* out, atdf_stream_t stream)
{
    if (!mlp_ok(mlp) || S < 0 || (S > 0 && (!x || !out))) return ATDF_ERR_INVALID_ARGUMENT;
    if (S == 0) return ATDF_OK;
    const cudaStream_t st = (cudaStream_t)stream;
    int sms = 0, optin = 0;
    if (const int e = device_limits(sms, optin)) return e;
    mlp::Plan p;
    const int i = pick_shape(kForward, *mlp, S, false, sms, optin, p);
    if (i >= 0) {
        auto fn = i == 0 ? mlp::forward_kernel<128, 8> : i == 1 ? mlp::forward_kernel<128, 4> : mlp::forward_kernel<128, 2>;
        return launch_tiles(fn, kForward[i], p, S, sms, st, *mlp, p, x, S, out);
    }
    mlp::row_forward_kernel<<<(unsigned)div_up(S, 128), 128, 0, st>>>(*mlp, x, S, out);
    ATDF_LAUNCH_CHECK();
    return ATDF_OK;
}

int atdf_mlp_backward(const atdf_mlp_t* mlp, const float* x, int64_t S, const float* grad_out, float* grad_x,
                      const atdf_mlp_grad_t* grad, atdf_stream_t stream)
{
    if (!mlp_ok(mlp) || !grad || S < 0 || (S > 0 && (!x || !grad_out))) return ATDF_ERR_INVALID_ARGUMENT;
    if (S == 0) return ATDF_OK;
    const cudaStream_t st = (cudaStream_t)stream;
    int sms = 0, optin = 0;
    if (const int e = device_limits(sms, optin)) return e;
    mlp::Plan p;
    const int i = pick_shape(kBackward, *mlp, S, true, sms, optin, p);
    if (i >= 0) {
        auto fn = i == 0   ? mlp::backward_kernel<128, 8>
                  : i == 1 ? mlp::backward_kernel<128, 4>
                  : i == 2 ? mlp::backward_kernel<256, 8>
                  : i == 3 ? mlp::backward_kernel<256, 4>
                           : mlp::backward_kernel<256, 2>;
        return launch_tiles(fn, kBackward[i], p, S, sms, st, *mlp, p, x, S, grad_out, grad_x, *grad);
    }
    mlp::row_backward_kernel<<<(unsigned)div_up(S, 64), 64, 0, st>>>(*mlp, x, S, grad_out, grad_x, *grad);
    ATDF_LAUNCH_CHECK();
    return ATDF_OK;
}

}  // extern "C"
